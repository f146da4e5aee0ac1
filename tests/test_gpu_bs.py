"""The ID's solve for small ranks, T = R11^-1 R12: the kernel with eight lanes a
column (few right-hand sides) and the one with a lane a column (many; the
rule lies at 64 right-hand sides an SM), at ranks around the row blocks of 8
and the largest rank.  A triangular solve's residual is within k roundings of
|R11| |T| in every entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 31, 33, 64, 127, 128])
def test_small_rank_solve(lra, dt, k):
    import torch
    rng = np.random.default_rng(k)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for nr, kernel in ((37, "trsm_bs_lanes_kernel"), (64 * sms + 33, "trsm_bs_kernel")):
        A = np.asfortranarray(rng.standard_normal((k + 2, k + nr)).astype(dt))
        o = lra.LRAOptions(dt, rank=k, rtol=0.0, sketch="none")
        ctx = lra.Context(0)
        V = lra.idfact(A, o, ctx=ctx)
        assert ctx.kernel_launches(kernel) == 1
        F = lra.pqrfact(A, o, ctx=ctx)
        ctx.close()
        assert V.k == F.k == k and np.array_equal(V.p, F.p)
        sel = np.unique(np.linspace(0, nr - 1, 64).astype(int))
        R11, R12 = F.R[:, :k].astype(np.longdouble), F.R[:, k:][:, sel].astype(np.longdouble)
        T = np.asarray(V.T)[:, sel].astype(np.longdouble)
        bound = (k + 4) * np.finfo(dt).eps * (np.abs(R11) @ np.abs(T))
        assert np.all(np.abs(R12 - R11 @ T) <= bound), (k, nr)
