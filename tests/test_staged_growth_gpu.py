"""Host products that go through page-locked memory take no device staging: as
their sizes rise, the lane allocates nothing and waits for nobody.  (Growing a
device buffer waits for all work on the device.)"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (10, 300, 3000, 7000, 16000)


def test_rising_sizes_wait_for_nobody(gpu):
    torch = pytest.importorskip("torch")
    side = torch.cuda.Stream()
    done = torch.cuda.Event()
    seen = {}

    def run():  # a thread of its own: a fresh lane
        rng = np.random.default_rng(1)
        x = torch.zeros(80000, dtype=torch.int64, device="cuda")
        # the lane's workspace and page-locked memory exist before
        gpu.mul_device(x.data_ptr(), 20000, x.data_ptr(), 20000, x.data_ptr() + 8 * 40000)
        gpu.stream_check()
        gpu.mul(np.ones(2, np.uint64), np.ones(2, np.uint64))
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(1_500_000_000)  # about 0.75 s of one SM
            done.record()
        for n in SIZES:
            a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for _ in range(2))
            got = gpu.mul(a, b)
            seen[n] = not done.query()
            x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
            assert got.tobytes() == x.to_bytes(16 * n, "little"), n

    for n in SIZES:  # the kernels are loaded (on this thread's lane)
        gpu.mul(np.ones(n, np.uint64), np.ones(n, np.uint64))
    t = threading.Thread(target=run)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert seen == {n: True for n in SIZES}
