"""The pivot exchange of the shared-memory QR (one word per CTA, read by a warp,
32 words a load): CTA counts on both sides of a load, and two requests at
once on SMs of their own.  No column's operations depend on the others of its
CTA, so every count gives the same bits."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(m, n, k, dt, seed):
    rng = np.random.default_rng(seed)
    A = (rng.standard_normal((m, k)) * 10.0 ** (-3.0 * np.arange(k) / k)) @ rng.standard_normal((k, n))
    A[:, n - 1] = A[:, 0]  # equal norms: the smaller index, whichever CTA has it
    return np.asfortranarray(A.astype(dt))


def _factor(lra, A, sms):
    ctx = lra.Context(0)
    ctx.set_tuning("qr_sms", 0, sms)
    F = lra.pqrfact(A, lra.LRAOptions(A.dtype.type, rtol=1e-5, precision="mixed", sketch="none"), ctx=ctx)
    assert ctx.kernel_launches("geqp3_df_smem_kernel" if A.dtype == np.float64 else "geqp3_f32_smem_kernel") == 1
    out = F.k, F.p.copy(), F.Q.copy(), F.R.copy()
    ctx.close()
    return out


def _same(a, b):
    return a[0] == b[0] and all(np.array_equal(x, y) for x, y in zip(a[1:], b[1:]))


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("m,n", [(72, 2400), (9, 1500)])
def test_cta_counts(lra, dt, m, n):
    A = _matrix(m, n, min(m, 50), dt, n)
    ref = _factor(lra, A, 0)
    assert ref[0] == min(m, 50)
    for sms in (8, 31, 32, 33, 64, 65, 96, 97, 128, 129):
        assert _same(_factor(lra, A, sms), ref), sms


def test_two_at_once(lra):
    mats = [_matrix(136, 900 + 37 * i, 100, np.float64, i) for i in range(4)]
    ref = [_factor(lra, A, 0) for A in mats]
    bad = []

    def work(t):
        try:
            for i in range(12):
                q = (i + t) % len(mats)
                if not _same(_factor(lra, mats[q], 60), ref[q]):
                    bad.append((t, i))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    ts = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad


def test_widest_sketches(lra):
    """As many columns as shared memory holds back to back, more than it holds an odd
    stride apart: the same factors, to the arithmetic, as with room to spare."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m, n = 40, 630 * sms  # 640 columns a CTA fit at a stride of 40 rows, 626 at 41
    rng = np.random.default_rng(2)
    A = np.asfortranarray(rng.standard_normal((m, n)) * 10.0 ** (-2.0 * rng.random(n)))
    ctx = lra.Context(0)
    o = lra.LRAOptions(rtol=1e-9, precision="mixed", sketch="none")
    F = lra.pqrfact(A, o, ctx=ctx)
    assert ctx.kernel_launches("geqp3_df_smem_kernel") == 1
    G = lra.pqrfact(np.asfortranarray(A[:, :600 * sms]), o, ctx=ctx)
    assert ctx.kernel_launches("geqp3_df_smem_kernel") == 2
    ctx.close()
    # pairs of floats: 2^-46 an operation, a column sees 40 steps
    for F, B in ((F, A), (G, A[:, :600 * sms])):
        assert F.k == m
        assert np.abs(B[:, F.p - 1] - F.Q @ F.R).max() <= m * 2.0 ** -46 * np.linalg.norm(A, axis=0).max()
        d = np.abs(np.diag(F.R[:, :m]))
        assert (d[1:] <= d[:-1] * (1 + 1e-6)).all()
