"""The double-float pivoted QR with its columns in global memory (the form
for sketches beyond shared memory, forced here by LRA_QR_SMEM=0) at the edges
of its schedule: fewer columns than CTAs, several columns a warp, a last row,
a rank that ends inside a block, norms recomputed inside a block, and a
reflector that leaves only one in shared memory."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = [(40, 7, 7, 1e-12), (33, 150, 33, 1e-12), (64, 153, 20, 1e-9), (300, 2500, 77, 1e-9), (1100, 1100, 500, 1e-9),
         (13000, 40, 40, 1e-9)]

CODE = """
import json, sys
sys.path.insert(0, {root!r}); sys.path.insert(0, {root!r} + "/lowrankapprox.jl_gb300")
import numpy as np
import lowrankapprox as lra
out = []
for m, n, k, rtol in {cases!r}:
    rng = np.random.default_rng(m + n)
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = np.linalg.qr(rng.standard_normal((n, k)))[0]
    s = 10.0 ** (-7.0 * np.arange(k) / max(k - 1, 1))
    A = np.asfortranarray((U * s) @ V.T)
    ctx = lra.Context(0)
    F = lra.pqrfact(A, lra.LRAOptions(rtol=rtol, precision="mixed", sketch="none"), ctx=ctx)
    E = A[:, F.p - 1] - F.Q @ F.R
    d = np.abs(np.diag(F.R[:, :F.k]))
    out.append([ctx.kernel_launches("geqp3_df_kernel"), F.k, float(np.linalg.norm(E)),
                float(np.abs(F.Q.T @ F.Q - np.eye(F.k)).max()), float((d[1:] / d[:-1]).max()) if F.k > 1 else 0.0])
    ctx.close()
print("RESULT " + json.dumps(out))
"""


def test_qr_global(lra):
    env = dict(os.environ, LRA_QR_SMEM="0")
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, cases=CASES)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:])
    for (m, n, k, rtol), (used, kk, err, orth, step) in zip(CASES, got):
        assert used == 1, (m, n)
        assert kk == k, (m, n, kk)
        # pairs of floats: 2^-46 an operation, at most m + k of them an entry
        assert err <= (m + k) * 2.0 ** -46, (m, n, err)
        assert orth <= (m + k) * 2.0 ** -46, (m, n, orth)
        # pivoting: |R_ii| does not grow beyond the norms' downdating error
        assert step <= 1.0 + 1e-6, (m, n, step)


def test_qr_global_many_columns(lra):
    """So many columns a CTA that only three pairs of each fit shared memory (as
    about a million do on all SMs): still in pairs of floats, with the factors
    that all SMs give."""
    code = CODE.replace("ctx = lra.Context(0)", "ctx = lra.Context(0); ctx.set_tuning('qr_sms', 0, sms)").replace(
        "for m, n, k, rtol in", "for sms, m, n, k, rtol in")
    cases = [(1, 40, 7000, 30, 1e-9), (1, 72, 8000, 40, 1e-9), (2, 300, 14000, 70, 1e-9)]
    r = subprocess.run([sys.executable, "-c", code.format(root=ROOT, cases=cases)], env=dict(os.environ, LRA_QR_SMEM="0"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:])
    for (_, m, n, k, rtol), (used, kk, err, orth, step) in zip(cases, got):
        assert used == 1, (m, n)
        assert kk == k, (m, n, kk)
        assert err <= (m + k) * 2.0 ** -46 and orth <= (m + k) * 2.0 ** -46, (m, n, err, orth)
        assert step <= 1.0 + 1e-6, (m, n, step)
