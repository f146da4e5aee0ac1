"""The limit of the bounded waits reaches every part of the library that
waits, and the waits between CTAs end by it: grid barriers and words that count
up in each part, the column exchange of the pivoted QRs.  Nothing sets what
the probes wait for; a part with a limit of its own would take 4 s."""
import time

import pytest

pytestmark = pytest.mark.gpu

WAITS = 6 * 2 + 2  # a barrier and a word in each of six parts, the exchange in two


def test_every_unit_has_the_limit(lra):
    from lowrankapprox import _ffi
    ctx = lra.Context(0)
    try:
        took = {}
        for ms in (1, 20):
            ctx.set_wait_limit(ms * 1_000_000)
            t0 = time.perf_counter()
            assert ctx.probe_wait() == _ffi.LRA_ETIMEDOUT, _ffi.load().lra_last_error(ctx.handle)
            took[ms] = time.perf_counter() - t0
        assert took[1] < 2.0
        assert WAITS * 0.020 <= took[20] < 4.0
    finally:
        ctx.set_wait_limit(0)
        ctx.close()
