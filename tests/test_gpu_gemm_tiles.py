"""The CUDA-core products at the edges of their tiles (8 x 16 and 32 x 32 for
FP64 and small FP32, 64 x 64), with and without split sums, plain and transposed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("m,n,order", [(1, 1, 1), (31, 15, 7), (33, 17, 9), (64, 33, 8), (1025, 65, 31), (2050, 16, 33),
                                       (300, 900, 640)])
def test_products(lra, dt, m, n, order):
    rng = np.random.default_rng(m)
    A = np.asfortranarray(rng.standard_normal((m, n)).astype(dt))
    for side, trans in (("left", "n"), ("left", "c"), ("right", "n"), ("right", "c")):
        op = (A if trans == "n" else A.T).astype(np.float64)
        M = op.shape[0] if side == "left" else op.shape[1]
        g = rng.standard_normal(order * M)
        B = lra.sketch(side, trans, A, order, lra.LRAOptions(dt, precision="native"), rand=lra.RandStream(gauss=g))
        if side == "left":
            S = g.reshape((order, M), order="F")
            R, scale = S @ op, np.abs(S) @ np.abs(op)
        else:
            S = g.reshape((M, order), order="F")
            R, scale = op @ S, np.abs(op) @ np.abs(S)
        # M terms summed in the type, and the draws rounded to it
        assert np.all(np.abs(B - R) <= (M + 4) * np.finfo(dt).eps * scale), (side, trans)
