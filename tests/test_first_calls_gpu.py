"""First calls of a process beside a busy stream: the kernels are loaded at start-up
(loading one waits for what the device is doing), so a first product of every
band returns while another stream is still at work."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, torch
from preclib_gb300 import native as N
N.init(0)
x = torch.from_numpy(np.random.default_rng(1).integers(0, 1 << 64, 1 << 20, dtype=np.uint64).view(np.int64)).cuda()
out = torch.empty(1 << 20, dtype=torch.int64, device="cuda")
# the thread's workspace and page-locked memory (growing them waits for the device)
N.mul_device(x.data_ptr(), 1 << 18, x.data_ptr(), 1 << 18, out.data_ptr())
N.mul(np.ones(1, np.uint64), np.ones(1, np.uint64))
N.stream_check()
side, done, late = torch.cuda.Stream(), torch.cuda.Event(), []
with torch.cuda.stream(side):
    torch.cuda._sleep(3_000_000_000)
    done.record()
for n in (40, 120, 200, 500, 1500, 3000, 6144):
    a = np.full(n, 3, np.uint64)
    q = int.from_bytes(a.tobytes(), "little") ** 2
    assert N.mul(a, a).tobytes() == q.to_bytes(16 * n, "little")
    late.append((n, done.query()))
s = torch.cuda.Stream()
for n in (64, 1500, 3000, 5000, 9000, 20000, 40000, 70000):
    N.mul_device(x.data_ptr(), n, x.data_ptr() + 8 * n, n, out.data_ptr(), s.cuda_stream)
    s.synchronize()
    late.append((n, done.query()))
print([n for n, d in late if d])
"""


def test_first_products_wait_for_nobody():
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == "[]", r.stdout
