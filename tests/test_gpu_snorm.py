"""The spectral norm's power iteration (one cooperative launch) against the
same iteration in numpy: sizes at the edges of its row blocks, column groups
and chunks, leading dimensions beyond the rows, the Hermitian form, and the
difference of two matrices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _power(D, x, herm, niter, rtol):
    D = D.astype(np.float64)
    x = x.astype(np.float64)
    nrm, s, t, it = np.linalg.norm(x), 1.0, 0.0, 0
    while s > 0 and abs(s - t) > t * rtol and it < niter:
        it += 1
        x = D @ (x / nrm)
        if not herm:
            x = D.T @ x
        nrm = np.linalg.norm(x)
        s, t = (nrm if herm else np.sqrt(nrm)), s
    return s


def _dev(A, pad):
    import torch
    m, n = A.shape
    buf = torch.zeros((n, m + pad), dtype=torch.from_numpy(A).dtype, device="cuda")
    V = buf.t()[:m]
    V.copy_(torch.from_numpy(A))
    return V


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("m,n,pad", [(1, 1, 0), (1, 301, 2), (300, 1, 0), (31, 33, 1), (257, 1000, 0), (5000, 67, 3),
                                     (64, 40000, 0), (1999, 1501, 5)])
def test_snorm_shapes(lra, dt, m, n, pad):
    rng = np.random.default_rng(m * 7 + n)
    A = rng.standard_normal((m, n)).astype(dt)
    B = (A + 1e-3 * rng.standard_normal((m, n))).astype(dt)
    x = rng.standard_normal(n)
    o = lra.LRAOptions(dt, rtol=0.0, snorm_niter=5)
    # every step's product sums at most m + n terms: a relative error of
    # (m + n) eps a step, entering the estimate of the last step only, as
    # the iteration corrects the direction's
    tol = 4 * (m + n) * np.finfo(dt).eps
    s = lra.snorm(_dev(A, pad), o, hermitian=False, rand=lra.RandStream(gauss=x))
    ref = _power(A, x, False, 5, 0.0)
    assert abs(s - ref) <= tol * ref
    d = lra.snormdiff(_dev(A, pad), _dev(B, pad + 1), o, rand=lra.RandStream(gauss=x))
    # A - B is rounded entry by entry: within the type's eps of |A - B|
    ref = _power(A.astype(np.float64) - B, x, False, 5, 0.0)
    assert abs(d - ref) <= (tol + 4 * np.sqrt(m * n) * np.finfo(dt).eps) * ref


@pytest.mark.parametrize("n", [1, 32, 97, 1200])
def test_snorm_hermitian(lra, n):
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n))
    A = A + A.T
    x = rng.standard_normal(n)
    o = lra.LRAOptions(rtol=0.0, snorm_niter=5)
    s = lra.snorm(_dev(A, 0), o, rand=lra.RandStream(gauss=x))
    ref = _power(A, x, True, 5, 0.0)
    assert abs(s - ref) <= 8 * n * np.finfo(float).eps * ref


def test_snorm_scales(lra):
    """Entries near the ends of the range neither overflow nor vanish in the
    norms; a zero matrix has norm zero."""
    rng = np.random.default_rng(3)
    A = rng.standard_normal((200, 130))
    x = rng.standard_normal(130)
    o = lra.LRAOptions(rtol=0.0, snorm_niter=4)
    for sc in (1e-120, 1e120):
        s = lra.snorm(_dev(A * sc, 0), o, rand=lra.RandStream(gauss=x))
        # the first step's change is judged against s = 1, as in the reference
        ref = _power(A, x, False, 4, 0.0) * sc
        assert abs(s - ref) <= 1e-12 * ref
    assert lra.snorm(_dev(A * 0, 0), o, rand=lra.RandStream(gauss=x)) == 0.0


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("m,n", [(31, 33), (33, 31), (257, 1000), (5000, 67), (64, 40000), (1999, 1501)])
def test_snorm_last_row_and_column(lra, dt, m, n):
    """A matrix whose norm sits in its last row, and in its last column: none of
    them is left out, in either type."""
    rng = np.random.default_rng(m + n)
    o = lra.LRAOptions(dt, rtol=0.0, snorm_niter=5)
    for last in (np.s_[m - 1, :], np.s_[:, n - 1]):
        A = 1e-3 * rng.standard_normal((m, n))
        A[last] += rng.standard_normal(A[last].shape)
        A = A.astype(dt)
        x = rng.standard_normal(n)
        ref = _power(A, x, False, 5, 0.0)
        assert abs(lra.snorm(_dev(A, 1), o, rand=lra.RandStream(gauss=x)) - ref) <= 4 * (m + n) * np.finfo(dt).eps * ref


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("m,n", [(40, 70), (70, 40), (3, 5000)])
def test_snorm_hermitian_flag_needs_a_square_matrix(lra, dt, m, n):
    """A rectangular matrix is not Hermitian, whatever the flag says."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((m, n)).astype(dt)
    o = lra.LRAOptions(dt, rtol=0.0, snorm_niter=5, seed=3)
    one, two = lra.Context(0), lra.Context(0)
    assert lra.snorm(A, o, hermitian=True, ctx=one) == lra.snorm(A, o, hermitian=False, ctx=two)
    one.close()
    two.close()
