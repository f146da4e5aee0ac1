"""The pivoted QR's conversions of a sketch to pairs of floats (done on the
bits of the entries) where their cases meet: entries that split exactly, ties
of the rounding, denormal low parts, zero and tiny columns, ranges that
underflow a sum of squares, and the batch's row- and column-major workspaces
against single calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _special(dt, seed):
    """60 x 90 matrices of full row rank with awkward entries."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((60, 90))
    out = {"plain": A}
    B = A.copy()
    B[:, 5] = 0
    B[:, 7] *= 1e-30
    out["tiny columns"] = B
    # 1 + j 2^-24 and one more bit: halfway cases of the 24-bit rounding
    C = 1.0 + rng.integers(0, 2 ** 10, (60, 90)) * 2.0 ** -24 + rng.integers(0, 2, (60, 90)) * 2.0 ** -52
    out["ties"] = C * rng.choice([-1.0, 1.0], (60, 90))
    out["powers"] = 2.0 ** rng.integers(-20, 1, (60, 90)) * rng.choice([-1.0, 1.0], (60, 90))
    out["small"] = A * (1e-280 if dt == np.float64 else 1e-30)
    return {k: np.asfortranarray(v.astype(dt)) for k, v in out.items()}


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_conversions(lra, dt):
    # pairs of floats resolve 2^-48 of the matrix's largest entry, FP32 2^-24;
    # a column sees 60 steps
    eps = 60 * (2.0 ** -46 if dt == np.float64 else 2.0 ** -22)
    for name, A in _special(dt, 7).items():
        F = lra.pqrfact(A, lra.LRAOptions(dt, rtol=0.0, precision="mixed", sketch="none"))
        A64 = A.astype(np.float64)
        sc = 1.0 / np.abs(A64).max()  # (numpy's norms underflow at the small case's scale)
        A64, R = A64 * sc, F.R.astype(np.float64) * sc
        E = A64[:, F.p - 1] - F.Q.astype(np.float64) @ R
        assert np.abs(E).max() <= eps * np.linalg.norm(A64, axis=0).max(), name
        # every pivot's norm is the largest of those left, to the arithmetic
        for i in range(F.k):
            left = np.linalg.norm(R[i:, i + 1:], axis=0)
            assert left.size == 0 or left.max() <= abs(R[i, i]) * (1 + 1e-5) + eps * abs(R[0, 0]), (name, i)


def test_batch_workspaces(lra):
    """Row-major (short sketches) and column-major (longer) workspaces give
    what single calls give."""
    import torch
    rng = np.random.default_rng(9)
    mats = []
    for m, n, k in [(100, 300, 10), (200, 31, 5), (64, 33, 30), (40, 65, 39), (500, 1030, 20), (900, 700, 150)]:
        A = rng.standard_normal((m, k)) @ rng.standard_normal((k, n))
        A[:, n // 2] = 0
        mats.append(torch.from_numpy(A).cuda().t().contiguous().t())
    o = lra.LRAOptions(rtol=1e-9, precision="mixed", seed=3)
    ctx = lra.Context(0)
    batch = lra.idfact_batched(mats, o, ctx=ctx)
    assert ctx.kernel_launches("df_finish_group_kernel") >= 1
    ctx.close()
    for A, V in zip(mats, batch):
        one = lra.Context(0)
        W = lra.idfact(A, o, ctx=one)
        one.close()
        assert np.array_equal(V.p, W.p) and np.array_equal(V.T, W.T)


def test_batch_long_rows(lra):
    """A raised qr_seq_len puts long sketches in the row-major workspace, also
    those whose tile of 32 columns no shared memory holds (order 1032)."""
    import torch
    rng = np.random.default_rng(4)
    mats = []
    for m, n, k in [(700, 1100, 560), (300, 200, 20)]:
        A = np.linalg.qr(rng.standard_normal((m, k)))[0] @ np.linalg.qr(rng.standard_normal((n, k)))[0].T
        mats.append(torch.from_numpy(A).cuda().t().contiguous().t())
    o = lra.LRAOptions(rtol=1e-9, precision="mixed", seed=3)

    def context():
        ctx = lra.Context(0)
        ctx.set_tuning("qr_seq_len", 0, 1200)
        return ctx

    ctx = context()
    batch = lra.idfact_batched(mats, o, ctx=ctx)
    assert ctx.kernel_launches("geqp3_df_group_kernel") >= 1
    ctx.close()
    for A, V in zip(mats, batch):
        one = context()
        W = lra.idfact(A, o, ctx=one)
        one.close()
        assert V.k == W.k and np.array_equal(V.p, W.p) and np.array_equal(V.T, W.T)


def test_conversions_to_pairs(lra):
    """The same for Float64 in pairs of floats (which a tolerance of zero does not
    take: the QR is then in FP64)."""
    eps = 60 * 2.0 ** -46
    ctx = lra.Context(0)
    for i, (name, A) in enumerate(_special(np.float64, 7).items()):
        F = lra.pqrfact(A, lra.LRAOptions(rtol=1e-13, precision="mixed", sketch="none"), ctx=ctx)
        assert ctx.kernel_launches("geqp3_df_smem_kernel") == i + 1, name
        sc = 1.0 / np.abs(A).max()
        A, R = A * sc, F.R * sc
        assert F.k == 60, name
        assert np.abs(A[:, F.p - 1] - F.Q @ R).max() <= eps * np.linalg.norm(A, axis=0).max(), name
        for j in range(F.k):
            left = np.linalg.norm(R[j:, j + 1:], axis=0)
            assert left.size == 0 or left.max() <= abs(R[j, j]) * (1 + 1e-5) + eps * abs(R[0, 0]), (name, j)
    ctx.close()
