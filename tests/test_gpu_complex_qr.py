"""The complex path's kernels at their edges: the pivoted QR with its columns in
shared memory against the general kernel (LRA_QR_SMEM=0; the same operations,
so the same bits), the solve by blocks of rows, and the product's tiles."""
import hashlib
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# rows, columns, rank, nb: one block and several, more columns than a warp each
# on all SMs, fewer rows than columns and the reverse
SHAPES = [(1, 1, 1, 32), (1, 9, 1, 32), (6, 1, 1, 32), (40, 7, 7, 32), (33, 150, 33, 8), (64, 153, 20, 1), (257, 1300, 60, 32),
          (300, 40, 25, 5), (1100, 90, 90, 32)]

CODE = """
import sys, json, hashlib
sys.path.insert(0, {root!r} + "/lowrankapprox.jl_gb300")
import numpy as np, torch
import lowrankapprox as lra
out = []
for dt in (np.complex128, np.complex64):
    for m, n, k, nb in {shapes!r}:
        for form in ("plain", "awkward", "nan", "allnan"):
            rng = np.random.default_rng(m + n)
            g = lambda a, b: rng.standard_normal((a, b)) + 1j * rng.standard_normal((a, b))
            A = (g(m, k) * 10.0 ** (-4 * np.arange(k) / k)) @ g(k, n)
            if form == "awkward":  # zero, equal, real, tiny and large columns
                A[:, n // 2] = 0
                A[:, n - 1] = A[:, 0]
                A[:, n // 3] = A[:, n // 3].real
                A[:, n // 4] *= 1e-30
                A *= 1e5
            if form == "nan":
                A[m // 2, n // 2] = np.nan
                A[0, n - 1] = np.inf
            if form == "allnan":
                A[:] = np.nan
            for rtol in (0.0, 1e-3):
                B = torch.from_numpy(np.ascontiguousarray(A.T.astype(dt))).cuda().t()
                ctx = lra.Context(0)
                jp, tau, kk = lra.geqp3_adap(B, lra.LRAOptions(dt, rtol=rtol, nb=nb, check_finite=False), ctx=ctx)
                h = hashlib.sha256(B.cpu().numpy().tobytes() + jp.cpu().numpy().tobytes() + tau[:kk].cpu().numpy().tobytes())
                out.append([str(np.dtype(dt)), m, n, form, rtol, kk, h.hexdigest(), ctx.kernel_launches("cgeqp3_smem_kernel")])
                ctx.close()
print("RESULT " + json.dumps(out))
"""


def test_qr_same_bits(lra):
    got = []
    for smem in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, shapes=SHAPES)],
                           env=dict(os.environ, LRA_QR_SMEM=smem), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:]))
    for a, b in zip(*got):
        assert a[7] == 1 and b[7] == 0, a
        if "nan" in a[3]:  # the payload of a NaN is nobody's
            assert a[:6] == b[:6], a
        else:
            assert a[:7] == b[:7], a


@pytest.mark.parametrize("dt", [np.complex128, np.complex64])
@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 127, 128, 129, 300])
def test_solve(lra, dt, k):
    rng = np.random.default_rng(k)
    n = k + 41
    A = np.asfortranarray((rng.standard_normal((k + 3, n)) + 1j * rng.standard_normal((k + 3, n))).astype(dt))
    o = lra.LRAOptions(dt, rank=k, rtol=0.0, sketch="none")
    V, F = lra.idfact(A, o), lra.pqrfact(A, o)
    assert V.k == F.k == k and np.array_equal(V.p, F.p)
    R11, R12, T = (np.asarray(x).astype(np.complex128) for x in (F.R[:, :k], F.R[:, k:], V.T))
    # a triangular solve's residual: k complex operations an entry, and R12 itself, which
    # the two calls hold to its rounding
    eps = 4 * (k + 4) * np.finfo(dt).eps
    bound = eps * (np.abs(R11) @ np.abs(T)) + eps * np.linalg.norm(A, axis=0).max()
    assert np.all(np.abs(R12 - R11 @ T) <= bound), k


@pytest.mark.parametrize("dt", [np.complex128, np.complex64])
@pytest.mark.parametrize("m,n,order", [(1, 1, 1), (31, 16, 8), (33, 17, 9), (64, 15, 7), (100, 33, 40), (257, 130, 72)])
def test_products(lra, dt, m, n, order):
    rng = np.random.default_rng(m)
    A = np.asfortranarray((rng.standard_normal((m, n)) + 1j * rng.standard_normal((m, n))).astype(dt))
    for side, trans in (("left", "n"), ("left", "c"), ("right", "n"), ("right", "c")):
        op = A.astype(np.complex128) if trans == "n" else A.astype(np.complex128).conj().T
        M = op.shape[0] if side == "left" else op.shape[1]
        g = rng.standard_normal(2 * order * M)
        z = g[0::2] + 1j * g[1::2]
        B = lra.sketch(side, trans, A, order, lra.LRAOptions(dt), rand=lra.RandStream(gauss=g))
        if side == "left":
            S = z.reshape((order, M), order="F")
            R, scale = S @ op, np.abs(S) @ np.abs(op)
        else:
            S = z.reshape((M, order), order="F")
            R, scale = op @ S, np.abs(op) @ np.abs(S)
        assert np.all(np.abs(B - R) <= 2 * (M + 4) * np.finfo(dt).eps * scale), (side, trans)
