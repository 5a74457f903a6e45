"""Device memory of a process that multiplies but never batches: the tables that
only batch classes read are made by the first batch that has such a class, for
its length, and not before."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, torch
from preclib_gb300 import native as N
torch.empty(1, device="cuda")
x = torch.from_numpy(np.random.default_rng(1).integers(0, 1 << 64, 2000 * 6000, dtype=np.uint64).view(np.int64)).cuda()
out = torch.empty_like(x)
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
N.init(0)
a = np.full(3000, 3, np.uint64)
want = int.from_bytes(a.tobytes(), "little") ** 2
assert N.mul(a, a).tobytes() == want.to_bytes(48000, "little")
N.mul_device(x.data_ptr(), 3000, x.data_ptr() + 24000, 3000, out.data_ptr())
N.stream_check()
print("start", (free0 - torch.cuda.mem_get_info()[0]) >> 20)
# 500 products of 2^14 points: a class with a table, in two batches
for count in (500, 2000):
    items = [(x.data_ptr() + 48000 * i, 3000, x.data_ptr() + 48000 * i + 24000, 3000, out.data_ptr() + 48000 * i)
             for i in range(count)]
    out.zero_()
    N.mul_batch(items)
    for i in (0, count - 1):
        p = x[6000 * i:6000 * i + 6000].cpu().numpy().tobytes()
        q = int.from_bytes(p[:24000], "little") * int.from_bytes(p[24000:], "little")
        assert out[6000 * i:6000 * i + 6000].cpu().numpy().tobytes() == q.to_bytes(48000, "little")
"""


def test_no_batch_tables_at_start():
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    # root and FP64 tables, one lane, and the kernels' code
    assert int(r.stdout.split()[1]) < 80, r.stdout
