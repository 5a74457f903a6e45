"""The library shut down and started again in one process: host, device and batch
products (direct, single-CTA and with twiddle tables) as before, and the memory
given back."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, torch
from preclib_gb300 import native as N
x = torch.from_numpy(np.random.default_rng(1).integers(0, 1 << 64, 6000 * 400, dtype=np.uint64).view(np.int64)).cuda()
out = torch.empty_like(x)

def exact(o, a, b):
    p = x[o:o + a + b].cpu().numpy().tobytes()
    q = int.from_bytes(p[:8 * a], "little") * int.from_bytes(p[8 * a:], "little")
    assert out[o:o + a + b].cpu().numpy().tobytes() == q.to_bytes(8 * (a + b), "little"), (o, a, b)

def everything():
    N.init(0)
    for n in (3, 300, 7000, 40000):
        a = np.full(n, 7, np.uint64)
        q = int.from_bytes(a.tobytes(), "little") ** 2
        assert N.mul(a, a).tobytes() == q.to_bytes(16 * n, "little")
    for an, bn in ((100, 90), (1500, 1400), (20000, 13000)):
        out.fill_(-1)
        N.mul_device(x.data_ptr(), an, x.data_ptr() + 8 * an, bn, out.data_ptr())
        N.stream_check()
        exact(0, an, bn)
    for an, bn in ((3000, 3000), (60, 60), (900, 800)):
        out.fill_(-1)
        N.mul_batch([(x.data_ptr() + 48000 * i, an, x.data_ptr() + 48000 * i + 8 * an, bn, out.data_ptr() + 48000 * i)
                     for i in range(400)])
        for i in (0, 399):
            exact(6000 * i, an, bn)

everything()
N.lib().prec_gpu_shutdown()
torch.cuda.synchronize()
free = []
for _ in range(3):
    everything()
    N.lib().prec_gpu_shutdown()
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
assert free[2] >= free[0] - (4 << 20), free
"""


def test_shutdown_and_start_again():
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
