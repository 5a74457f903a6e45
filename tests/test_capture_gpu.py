"""Device products captured into the caller's own graph: one of up to 2^12
points uses no memory of the calling thread's lane, so it is accepted whatever
the thread multiplied before, and its replays stay exact while the thread makes
other products (which move the lane's workspace)."""
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(a, b):
    x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
    return np.frombuffer(x.to_bytes(8 * (len(a) + len(b)), "little"), dtype=np.uint64)


@pytest.mark.parametrize("an,bn", [(1, 1), (64, 50), (1000, 24), (1024, 1024)])
def test_small_product_in_a_graph(gpu, an, bn):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(an)
    dev = lambda x: torch.from_numpy(x.view(np.int64)).cuda()  # noqa: E731
    a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for n in (an, bn))
    ta, tb = dev(a), dev(b)
    out = torch.zeros(an + bn, dtype=torch.int64, device="cuda")
    s = torch.cuda.Stream()
    other = dev(rng.integers(0, 1 << 64, 1 << 20, dtype=np.uint64))
    big = torch.empty(1 << 21, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    gpu.mul_device(ta.data_ptr(), an, tb.data_ptr(), bn, out.data_ptr(), s.cuda_stream)  # the lane is in use
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        gpu.mul_device(ta.data_ptr(), an, tb.data_ptr(), bn, out.data_ptr(), s.cuda_stream)
    for rep in range(3):
        a = rng.integers(0, 1 << 64, an, dtype=np.uint64)
        ta.copy_(torch.from_numpy(a.view(np.int64)))
        out.zero_()
        torch.cuda.synchronize()
        # a direct product and one that grows the workspace, on another stream
        n = 3000 << (2 * rep)
        gpu.mul_device(other.data_ptr(), 1000, other.data_ptr(), 900, big.data_ptr())
        gpu.mul_device(other.data_ptr(), n, other.data_ptr(), n, big.data_ptr())
        with torch.cuda.stream(s):
            graph.replay()
        gpu.mul_device(other.data_ptr(), 1000, other.data_ptr(), 900, big.data_ptr())
        gpu.stream_check()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint64), _exact(a, b)), rep
        want = _exact(other[:1000].cpu().numpy(), other[:900].cpu().numpy())
        assert np.array_equal(big[:1900].cpu().numpy().view(np.uint64), want), rep


@pytest.mark.parametrize("an,bn", [(1000, 24), (3000, 2500), (40000, 25536)])
def test_noalloc_product_in_a_graph(gpu, an, bn):
    """The no-allocation entry point at every kind of length it takes."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(an)
    L = gpu.lib()
    out = torch.zeros(an + bn, dtype=torch.int64, device="cuda")
    ta = torch.zeros(an, dtype=torch.int64, device="cuda")
    b = rng.integers(0, 1 << 64, bn, dtype=np.uint64)
    tb = torch.from_numpy(b.view(np.int64)).cuda()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    args = (ta.data_ptr(), an, tb.data_ptr(), bn, out.data_ptr(), s.cuda_stream)
    gpu.check(L.prec_gpu_mul_device_noalloc(*args))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        gpu.check(L.prec_gpu_mul_device_noalloc(*args))
    for rep in range(2):
        a = rng.integers(0, 1 << 64, an, dtype=np.uint64)
        ta.copy_(torch.from_numpy(a.view(np.int64)))
        out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            graph.replay()
        gpu.stream_check(s.cuda_stream)
        assert np.array_equal(out.cpu().numpy().view(np.uint64), _exact(a, b)), rep


LONGER = """
import numpy as np, torch
from preclib_gb300 import native as N
N.init(0)
z = np.zeros(1, np.uint64)
N.mul(z, z)  # the thread's lane, without a product on it
rng = np.random.default_rng(1)
a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for n in (1500, 1400))
ta, tb = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
out = torch.zeros(2900, dtype=torch.int64, device="cuda")
s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
torch.cuda.synchronize()
n0 = N.launch_count()
with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
    N.mul_device(ta.data_ptr(), 1500, tb.data_ptr(), 1400, out.data_ptr(), s.cuda_stream)
print(N.launch_count() - n0)
g.replay()
torch.cuda.synchronize()
x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
assert out.cpu().numpy().tobytes() == x.to_bytes(8 * 2900, "little")
"""


def test_longer_product_in_a_graph():
    """Four-step kernels, not the direct one, whose counter is the lane's."""
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", LONGER], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout) == 4
