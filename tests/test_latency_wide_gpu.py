"""The kernels of single products of 2^18 points on 64-bit digits (131073 .. 262144
limbs in all), on the device: every number of eighths they keep at its shortest
and longest products, balanced, uneven (one operand as long as the plan takes) and
squares, random and all-ones limbs, with guards around the result, against the
oracle."""
import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu

HALF = 1 << 17  # the longest operand


@pytest.mark.parametrize("total", [HALF + 2] + [n for e in (5, 6, 7) for n in ((e << 15) + 1, (e << 15) + 2)] + [2 * HALF])
def test_eighths(gpu, total):
    torch = pytest.importorskip("torch")
    for an, pattern in ((total // 2, "random"), (total // 2, "ones"), (min(HALF, total - total // 5), "random"),
                        (min(HALF, total - 40), "ones"), (total // 2, "square")):
        bn = total - an
        if pattern == "square":
            bn = an
            if 2 * an < HALF + 2:
                continue
        assert gpu.ntt_log2(an, bn) == 18  # 64-bit digits: on 32-bit digits this length is 2^19
        a, b = O.splitmix64(an, an), O.splitmix64(bn + 1, bn)
        if pattern == "ones":
            a[:], b[:] = ~np.uint64(0), ~np.uint64(0)
        ta, tb = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
        if pattern == "square":
            b, tb = a, ta
        to = torch.full((an + bn + 2,), -7, dtype=torch.int64, device="cuda")
        gpu.mul_device(ta.data_ptr(), an, tb.data_ptr(), bn, to.data_ptr() + 8)
        gpu.stream_check()
        got = to.cpu().numpy()
        assert got[0] == got[-1] == -7
        assert np.array_equal(got[1:-1].view(np.uint64), O.mul_ntt(a, b)), (an, bn, pattern)


def test_the_digits(gpu):
    prev = gpu.set_wide_digits(False)
    try:
        assert gpu.ntt_log2(HALF, HALF) == 19
    finally:
        gpu.set_wide_digits(prev)
    a = O.splitmix64(1, HALF)
    gpu.mul(a, a[: HALF // 2])
    st = gpu.last_stats()
    assert (st.log2_n, st.digit_bits, st.primes) == (18, 64, 5)
