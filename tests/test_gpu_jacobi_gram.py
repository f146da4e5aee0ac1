"""The FP32 sweeps on Gram products (jacobi_gram.cu) that precede the polish
of psvdfact's core SVD on the mixed path, at core orders on both sides of
its edges: one pair of 32-column blocks, odd and even block counts, a last
block of one column, several row tiles per CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(m, n, k, seed):
    """Numerical rank k, singular values from 1 to 1e-9."""
    rng = np.random.default_rng(seed)
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = np.linalg.qr(rng.standard_normal((n, k)))[0]
    s = 10.0 ** (-9.0 * np.arange(k) / max(k - 1, 1))
    return (U * s) @ V.T, s


@pytest.mark.parametrize("k", [64, 65, 95, 96, 97, 128, 160, 161, 193, 449, 640, 2050])
def test_gram_sweeps(lra, k):
    m, n = k + 300, k + 150
    A, s = _matrix(m, n, k, k)
    ctx = lra.Context(0)
    F = lra.psvdfact(A, lra.LRAOptions(rtol=1e-10, precision="mixed", seed=3), ctx=ctx)
    used = ctx.kernel_launches("jacobi_gram_kernel")
    ctx.close()
    assert used == 1
    assert F.k == k
    # absolute accuracy of the mixed path: 2^-48 of the sketch and 2^-45 of
    # its GEMMs, times the order's growth: well below 1e-11 of s_1
    assert np.abs(F.S - s).max() <= 1e-11
    U, Vt = np.asarray(F.U), np.asarray(F.Vt)
    assert np.linalg.norm(A - (U * F.S) @ Vt) <= 1e-10
    for Q in (U, Vt.T):
        assert np.abs(Q.T @ Q - np.eye(k)).max() < 1e-10


def test_gram_sweeps_clusters(lra):
    """Equal singular values (no gaps to separate): the same singular values,
    and factors no further from orthonormal than after the in-cluster sweeps
    (both are finished by the pairwise sweeps, run to their last cosine)."""
    rng = np.random.default_rng(8)
    U = np.linalg.qr(rng.standard_normal((400, 90)))[0]
    V = np.linalg.qr(rng.standard_normal((300, 90)))[0]
    s = np.repeat([1.0, 1e-3, 1e-6], 30)
    A = (U * s) @ V.T
    defect = []
    for cluster in (-1, 0):
        ctx = lra.Context(0)
        ctx.set_tuning("jacobi_cluster", 0, cluster)
        F = lra.psvdfact(A, lra.LRAOptions(rtol=1e-8, precision="mixed", seed=3), ctx=ctx)
        assert ctx.kernel_launches("jacobi_gram_kernel") == (1 if cluster < 0 else 0)
        ctx.close()
        assert F.k == 90
        assert np.abs(F.S - s).max() <= 1e-11
        defect.append(max(np.abs(Q.T @ Q - np.eye(90)).max() for Q in (np.asarray(F.U), np.asarray(F.Vt).T)))
    assert defect[0] <= 4 * defect[1] + 1e-10


def test_gram_sweeps_beside_another_request(lra):
    """Two requests at once, each with the other's kernels on its SMs: the CTAs of
    a pair of blocks take the same rotations however far apart they run, so
    both give the bits of a call alone."""
    import threading
    mats = [_matrix(k + 300, k + 150, k, k)[0] for k in (449, 640, 385)]

    def run(A):
        ctx = lra.Context(0)
        F = lra.psvdfact(A, lra.LRAOptions(rtol=1e-10, precision="mixed", seed=3), ctx=ctx)
        assert ctx.kernel_launches("jacobi_gram_kernel") == 1
        out = [np.array(F.U), np.array(F.S), np.array(F.Vt)]
        ctx.close()
        return out

    ref = [run(A) for A in mats]
    bad = []

    def work(t):
        try:
            for i in range(9):
                q = (i + t) % len(mats)
                if not all(np.array_equal(x, y) for x, y in zip(run(mats[q]), ref[q])):
                    bad.append((t, i))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    ts = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
