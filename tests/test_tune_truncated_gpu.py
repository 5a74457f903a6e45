"""A tuned length keeps its truncated transforms: after the autotuner has gone
over the lengths of 2^20 .. 2^22 points, products that need five or six eighths
take no longer than with the default configuration (a candidate that is 1% faster
on whole transforms only, and without truncated kernels, makes them 20 - 40% slower)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _times(gpu, torch, x, out, sizes):
    """Best of 15, L2 flushed before each."""
    flush = torch.empty(1 << 26, dtype=torch.int32, device="cuda")
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    r = []
    for n in sizes:
        best = float("inf")
        for _ in range(15):
            flush.zero_()
            start.record()
            gpu.mul_device(x.data_ptr(), n, x.data_ptr() + 8 * (1 << 20), n, out.data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        r.append(best)
    return r


def test_tuned_lengths_keep_truncated_products(gpu):
    torch = pytest.importorskip("torch")
    x = torch.from_numpy(np.random.default_rng(2).integers(0, 1 << 64, 1 << 21, dtype=np.uint64).view(np.int64)).cuda()
    out = torch.empty(1 << 21, dtype=torch.int64, device="cuda")
    sizes = [e << (k - 5) for k in (20, 21, 22) for e in (5, 6)]
    prev = gpu.set_wide_digits(False)  # tables are tuned on 32-bit digits
    gpu.tune_reset()
    try:
        _times(gpu, torch, x, out, sizes)
        before = _times(gpu, torch, x, out, sizes)
        gpu.autotune(20, 22)
        after = _times(gpu, torch, x, out, sizes)
    finally:
        gpu.tune_reset()
        gpu.set_wide_digits(prev)
    for n, b, a in zip(sizes, before, after):
        assert a < 1.12 * b, (n, b, a)
