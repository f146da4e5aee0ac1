"""Cholesky and triangular inverse at the edges of their blocks of 32, through
psvd's factors: ranks around 32, 64, 96, ... on both types; the factors are
orthonormal and reproduce the matrix, which a wrong block would not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 65, 95, 96, 97, 130, 257, 290, 515, 600])
def test_psvd_ranks(lra, dt, k):
    rng = np.random.default_rng(k)
    U, V = np.linalg.qr(rng.standard_normal((k + 700, k)))[0], np.linalg.qr(rng.standard_normal((k + 650, k)))[0]
    s = 10.0 ** (-2.0 * np.arange(k) / k)
    A = (U * s) @ V.T
    rtol = 1e-9 if dt == np.float64 else 1e-4
    F = lra.psvdfact(np.asfortranarray(A.astype(dt)), lra.LRAOptions(dt, rtol=rtol, precision="mixed"))
    assert F.k == k
    # two orders above the type's (mixed path's) rounding of a k-term product
    tol = 100 * np.sqrt(k) * (2.0 ** -42 if dt == np.float64 else 2.0 ** -22)
    U1, V1 = F.U.astype(np.float64), F.Vt.astype(np.float64)
    assert np.abs(U1.T @ U1 - np.eye(k)).max() <= tol and np.abs(V1 @ V1.T - np.eye(k)).max() <= tol
    assert np.abs(F.S - s).max() <= tol
    assert np.abs((U1 * F.S.astype(np.float64)) @ V1 - A).max() <= tol
