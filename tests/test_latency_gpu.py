"""The kernels of single products of 2^13 .. 2^18 points, on the device: every
length at its shortest and longest products, uneven operands (one past half
the transform) and squares, with carries through every limb, against the
oracle."""
import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", (True, False))
@pytest.mark.parametrize("k", range(13, 19))
def test_lengths(gpu, k, wide):
    torch = pytest.importorskip("torch")
    prev = gpu.set_wide_digits(wide)
    try:
        top = 1 << (k - 1)  # limbs of the longest product
        for total in (top // 2 + 2, top * 5 // 8, top * 3 // 4 + 1, top):
            if total * total // 4 <= 1 << 22:  # formed directly
                continue
            for an in (total // 2, total - total // 3, total - 40):
                bn = total - an
                if an * bn <= 1 << 22 and an <= 4096:
                    continue
                for pattern in ("random", "ones"):
                    a, b = O.splitmix64(an, an), O.splitmix64(bn + 1, bn)
                    if pattern == "ones":
                        a[:], b[:] = ~np.uint64(0), ~np.uint64(0)
                    ta, tb = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
                    to = torch.full((total + 2,), -7, dtype=torch.int64, device="cuda")
                    gpu.mul_device(ta.data_ptr(), an, tb.data_ptr(), bn, to.data_ptr() + 8)
                    gpu.stream_check()
                    got = to.cpu().numpy()
                    assert got[0] == got[-1] == -7
                    assert np.array_equal(got[1:-1].view(np.uint64), O.mul_ntt(a, b)), (an, bn, pattern)
                    if an == total // 2:
                        to = torch.full((2 * an,), -7, dtype=torch.int64, device="cuda")
                        gpu.mul_device(ta.data_ptr(), an, ta.data_ptr(), an, to.data_ptr())
                        gpu.stream_check()
                        assert np.array_equal(to.cpu().numpy().view(np.uint64), O.mul_ntt(a, a)), (an, pattern)
    finally:
        gpu.set_wide_digits(prev)
