"""A batch's pivoted QRs by gangs of blocks in shared memory: one matrix (a
gang as wide as it may be), fewer and more matrices than blocks, odd shapes,
columns short and long, sketches at ranks that end at different steps.  The
kernel with the columns in global memory (LRA_QR_SMEM=0) runs the same
arithmetic, so both give the same bits."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# (matrices, rows, columns, rank)
BATCHES = [(1, 300, 500, 12), (3, 65, 33, 30), (7, 513, 1031, 70), (40, 128, 257, 1), (200, 96, 64, 20)]

CODE = """
import sys, json, hashlib
sys.path.insert(0, {root!r})
sys.path.insert(0, {root!r} + "/lowrankapprox.jl_gb300")
import numpy as np, torch
import lowrankapprox as lra
out = []
for c, m, n, k in {batches!r}:
    rng = np.random.default_rng(m + c)
    mats = []
    for i in range(c):
        r = max(1, k - i % 7)
        A = rng.standard_normal((m, r)) @ rng.standard_normal((r, n - i % 3))
        mats.append(torch.from_numpy(np.ascontiguousarray(A.T)).cuda().t())
    ctx = lra.Context(0)
    res = lra.idfact_batched(mats, lra.LRAOptions(rtol=1e-9, precision="mixed", seed=5), ctx=ctx)
    h = hashlib.sha256()
    for V in res:
        h.update(np.ascontiguousarray(V.p).tobytes() + np.ascontiguousarray(V.T).tobytes())
    out.append([ctx.kernel_launches("geqp3_df_gang_kernel"), ctx.kernel_launches("geqp3_df_group_kernel"),
                [V.k for V in res], h.hexdigest()])
    ctx.close()
print("RESULT " + json.dumps(out))
"""


def test_gangs(lra):
    got = []
    for smem in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, batches=BATCHES)],
                           env=dict(os.environ, LRA_QR_SMEM=smem), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(json.loads([x for x in r.stdout.splitlines() if x.startswith("RESULT ")][0][7:]))
    for (c, m, n, k), a, b in zip(BATCHES, *got):
        assert a[0] >= 1 and a[1] == 0, (c, a[:2])
        assert b[0] == 0 and b[1] >= 1, (c, b[:2])
        assert a[2] == [max(1, k - i % 7) for i in range(c)], c
        assert a[2:] == b[2:], (c, m, n)
