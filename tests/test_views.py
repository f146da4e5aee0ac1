"""numpy views of library results: column-major, writable, and the result freed
when the last view is gone, not before."""
import ctypes
import gc

import numpy as np
import lowrankapprox as L


def test_result_views():
    freed = []
    mem = (ctypes.c_double * 12)(*range(12))
    own = L._Result(freed.append, "r")
    a = L._view(ctypes.addressof(mem), (3, 2), np.float64, own)
    b = L._view(ctypes.addressof(mem) + 48, (6,), np.int64, own)
    z = L._view(0, (0, 4), np.float32, own)
    assert a.flags.f_contiguous and a.flags.writeable and np.array_equal(a, [[0, 3], [1, 4], [2, 5]])
    assert b.dtype == np.int64 and b.shape == (6,) and np.array_equal(b.view(np.float64), np.arange(6, 12))
    assert z.shape == (0, 4) and z.dtype == np.float32
    a[1, 1] = 40
    assert mem[4] == 40
    del own, a
    gc.collect()
    assert not freed
    tail = b[4:]
    del b
    gc.collect()
    assert not freed
    del tail
    gc.collect()
    assert freed == ["r"]
