"""The FP64 pivoted QR with its columns in shared memory against the one that
keeps them in global memory (LRA_QR_SMEM=0): the same operations, so the same
bits, for one block and several, more columns than warps, zero, equal, tiny
and large columns, ranks that end inside a block of pivots, and inputs that are
not finite."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(1, 1, 1, 32), (1, 9, 1, 32), (6, 1, 1, 32), (40, 7, 7, 32), (33, 150, 33, 8), (64, 153, 20, 1), (257, 2600, 60, 32),
          (300, 40, 25, 5), (1100, 90, 90, 32)]

CODE = """
import sys, json, hashlib
sys.path.insert(0, {root!r} + "/lowrankapprox.jl_gb300")
import numpy as np, torch
import lowrankapprox as lra
out = []
for m, n, k, nb in {shapes!r}:
    for form in ("plain", "awkward", "small", "nan", "allnan"):
        rng = np.random.default_rng(m + n)
        A = (rng.standard_normal((m, k)) * 10.0 ** (-4 * np.arange(k) / k)) @ rng.standard_normal((k, n))
        if form == "awkward":
            A[:, n // 2] = 0
            A[:, n - 1] = A[:, 0]
            A[:, n // 4] *= 1e-30
            A *= 1e5
        if form == "small":
            A *= 1e-300
        if form == "nan":
            A[m // 2, n // 2] = np.nan
            A[0, n - 1] = np.inf
        if form == "allnan":
            A[:] = np.nan
        for rtol in (0.0, 1e-3):
            B = torch.from_numpy(A.T.copy()).cuda().t()
            ctx = lra.Context(0)
            jp, tau, kk = lra.geqp3_adap(B, lra.LRAOptions(rtol=rtol, nb=nb, check_finite=False), ctx=ctx)
            h = hashlib.sha256(B.cpu().numpy().tobytes() + tau[:kk].cpu().numpy().tobytes()).hexdigest()
            p = hashlib.sha256(jp.cpu().numpy().tobytes()).hexdigest()
            out.append([m, n, form, rtol, kk, p, h, ctx.kernel_launches("geqp3_f64_smem_kernel")])
            ctx.close()
print("RESULT " + json.dumps(out))
"""


def test_same_bits(lra):
    got = []
    for smem in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, shapes=SHAPES)],
                           env=dict(os.environ, LRA_QR_SMEM=smem), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:]))
    for a, b in zip(*got):
        assert a[7] == 1 and b[7] == 0, a
        # (the payload of a NaN is nobody's)
        assert a[:6] == b[:6] and ("nan" in a[2] or a[6] == b[6]), (a, b)


def test_tall_sketches_spread_over_all_blocks(lra):
    """Columns too long for eight a block: they are spread over every block, and
    stay in shared memory."""
    code = CODE.replace('("plain", "awkward", "small", "nan", "allnan")', '("plain", "awkward", "nan")')
    got = []
    for smem in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", code.format(root=ROOT, shapes=[(4000, 300, 90, 32), (3600, 200, 40, 32)])],
                           env=dict(os.environ, LRA_QR_SMEM=smem), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:]))
    for a, b in zip(*got):
        assert a[7] == 1 and b[7] == 0, a
        assert a[:6] == b[:6] and ("nan" in a[2] or a[6] == b[6]), (a, b)
