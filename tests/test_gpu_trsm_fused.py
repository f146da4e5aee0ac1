"""The Float32 solve in one launch (up to rank 1024 and 32 right-hand sides an SM)
and the recursion beyond, at ranks around blocks of 32 and halves: the residual
of T = R11^-1 R12 is within rank roundings of |R11| |T| in every entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [129, 160, 161, 193, 257, 500, 1000, 1024, 1025])
def test_solve(lra, k):
    import torch
    rng = np.random.default_rng(k)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for nr in (1, 37) + ((32 * sms, 32 * sms + 1) if k in (129, 193) else ()):
        A = np.asfortranarray(rng.standard_normal((k + 2, k + nr)).astype(np.float32))
        o = lra.LRAOptions(np.float32, rank=k, rtol=0.0, sketch="none")
        ctx = lra.Context(0)
        V = lra.idfact(A, o, ctx=ctx)
        # (a larger rank's halves are solved so)
        assert ctx.kernel_launches("trsm_fused_kernel") == (0 if nr > 32 * sms else 1 if k <= 1024 else 2)
        F = lra.pqrfact(A, o, ctx=ctx)
        ctx.close()
        assert V.k == F.k == k and np.array_equal(V.p, F.p)
        sel = np.unique(np.linspace(0, nr - 1, 64).astype(int))
        R11, R12 = F.R[:, :k].astype(np.float64), F.R[:, k:][:, sel].astype(np.float64)
        T = np.asarray(V.T)[:, sel].astype(np.float64)
        assert np.all(np.abs(R12 - R11 @ T) <= (k + 8) * np.finfo(np.float32).eps * (np.abs(R11) @ np.abs(T) + np.abs(R12))), nr
