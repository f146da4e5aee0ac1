"""The tensor-core sketch's operand written straight from its draws: the
injected stream and the library generator, left and right layouts, both types,
orders around the tile heights and odd lengths.  Numbers on the lattice are
exact in both, so a sketch with the generator equals one with its draws
injected bit for bit, and a right sketch of A the transpose of a left sketch
of A' with the stream's matrix transposed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# order 1, edges of tiles of 96 and 128 rows, odd numbers of draws, M around
# chunks of 64 and 512
CASES = [(1, 33, 5), (7, 63, 40), (96, 65, 130), (97, 513, 64), (128, 511, 129), (129, 1031, 37), (257, 200, 300)]


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("order,m,n", CASES)
def test_sources(lra, dt, order, m, n):
    rng = np.random.default_rng(order + m)
    A = np.asfortranarray(rng.standard_normal((m, n)).astype(dt))
    o = lra.LRAOptions(dt, precision="mixed", seed=11)
    for side, trans, M in (("left", "n", m), ("left", "c", n), ("right", "n", n), ("right", "c", m)):
        ctx = lra.Context(0)
        own = lra.sketch(side, trans, A, order, o, ctx=ctx)
        g = lra.library_gauss(11, order * M)
        given = lra.sketch(side, trans, A, order, o, ctx=ctx, rand=lra.RandStream(gauss=g))
        ctx.close()
        assert np.array_equal(own, given), (side, trans)
        op = (A if trans == "n" else A.T).astype(np.float64)
        if side == "left":
            S = g.reshape((order, M), order="F")
            R, scale = S @ op, np.abs(S).sum(1)[:, None] * np.abs(op).max(0)[None, :]
        else:
            S = g.reshape((M, order), order="F")
            R, scale = op @ S, np.abs(op).max(1)[:, None] * np.abs(S).sum(0)[None, :]
        # columns truncated at 2^-48 (Float32: 2^-24) of their scale, and the result's rounding
        tol = 2.0 ** -46 if dt == np.float64 else 2.0 ** -22
        assert np.all(np.abs(given - R) <= tol * scale + 4 * np.finfo(dt).eps * np.abs(R)), (side, trans)
        if side == "right":
            T = lra.sketch("left", "n" if trans == "c" else "c", A, order, o,
                           rand=lra.RandStream(gauss=np.ascontiguousarray(S).ravel()))
            assert np.array_equal(given, T.T), trans
