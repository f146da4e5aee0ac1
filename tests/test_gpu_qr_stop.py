"""Adaptive steps end their QR once the rank has reached the step's threshold
(32, 64, ...): ranks around the thresholds give the rank, and as many steps as the
doubling loop takes (k < 32 2^t ends it), on every path that has the stop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(k, dt, seed):
    rng = np.random.default_rng(seed)
    def g(m, n):
        A = rng.standard_normal((m, n))
        return A + 1j * rng.standard_normal((m, n)) if np.issubdtype(dt, np.complexfloating) else A
    U, V = np.linalg.qr(g(300, k))[0], np.linalg.qr(g(400, k))[0]
    return np.asfortranarray(((U * 2.0 ** (-np.arange(k) / 16)) @ V.conj().T).astype(dt))


@pytest.mark.parametrize("k", [1, 31, 32, 33, 40, 41, 63, 64, 65, 128])
@pytest.mark.parametrize("dt,precision", [(np.float64, "mixed"), (np.float64, "native"), (np.float32, "mixed"),
                                          (np.complex128, "native"), (np.complex64, "native")])
def test_ranks_at_thresholds(lra, dt, precision, k):
    A = _matrix(k, dt, k)
    V = lra.idfact(A, lra.LRAOptions(dt, rtol=1e-4, precision=precision, seed=7))
    assert V.k == k
    assert V.nsteps == 1 + next(t for t in range(9) if k < 32 * 2 ** t)
    E = A[:, V.rd - 1] - A[:, V.sk - 1] @ V.T
    assert np.abs(E).max() <= 1e-3 * np.abs(A).max()


def test_batch(lra):
    ranks = [1, 31, 32, 33, 64, 65, 128]
    o = lra.LRAOptions(rtol=1e-4, precision="mixed", seed=7)
    for k, V in zip(ranks, lra.idfact_batched([_matrix(k, np.float64, k) for k in ranks], o)):
        assert V.k == k and V.nsteps == 1 + next(t for t in range(9) if k < 32 * 2 ** t)


CODE = """
import sys
sys.path.insert(0, {root!r} + "/lowrankapprox.jl_gb300"); sys.path.insert(0, {root!r} + "/tests")
import numpy as np
import lowrankapprox as lra
from test_gpu_qr_stop import _matrix
dt = np.{dt}
A = _matrix(100, dt, 100)
o = lra.LRAOptions(dt, rtol=1e-4, precision={precision!r}, seed=7)
V = lra.idfact_batched([A, A[:, :350].copy(order="F")], o)[0] if {batch} else lra.idfact(A, o)
assert V.k == 100
"""


@pytest.mark.parametrize("dt,precision,batch", [("float64", "mixed", 0), ("float64", "native", 0), ("float32", "mixed", 0),
                                                ("complex128", "native", 0), ("complex64", "native", 0),
                                                ("float64", "mixed", 1)])
def test_steps_end_at_their_thresholds(lra, dt, precision, batch):
    """A matrix of rank 100: the QRs of orders 40 and 72 end with 32 and 64 pivots
    (without the early end they would go on to 40 and 72), that of 136 reveals
    the rank."""
    import os
    import re
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE.format(root=root, dt=dt, precision=precision, batch=batch)],
                       env=dict(os.environ, LRA_TRACE="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    steps = re.findall(r"step of order (\d+), threshold (\d+): rank (-?\d+)", r.stderr)
    assert set(steps) == {("40", "32", "32"), ("72", "64", "64"), ("136", "128", "100")}, steps
    assert len(steps) == 3 * (1 + batch)
