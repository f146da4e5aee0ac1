"""The double-float Jacobi sweeps where their shapes change: orders around a
block of columns, odd and even numbers of blocks, the rows a lane holds (128,
256, 512), on a core whose singular values are all equal, where they run to
the last cosine."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 12, 13, 127, 128, 129, 255, 257, 511, 512])
def test_df_sweeps(lra, n):
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n + 20, n)))
    P, _ = np.linalg.qr(rng.standard_normal((n + 30, n)))
    o = lra.LRAOptions(rtol=1e-10, precision="mixed", sketch="none")
    # the sweeps leave cosines of a few 2^-46 sqrt(n); the factors around them
    # are of the same precision
    tol = 64 * np.sqrt(n + 30) * 2.0 ** -46 * np.sqrt(n)
    F = lra.psvdfact(np.asfortranarray(Q @ P.T), o)
    assert F.k == n and np.abs(F.S - 1).max() <= tol
    assert np.abs(F.U.T @ F.U - np.eye(n)).max() <= tol and np.abs(F.Vt @ F.Vt.T - np.eye(n)).max() <= tol
