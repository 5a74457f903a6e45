"""GPU tests of host products whose kernels overlap with their copies (from 2^19
points, one launch per pass on a side stream below 2^21): the sizes around
the edges of 2^18 .. 2^21 points for both digit widths, a square, the result
over an operand and two threads at once; each equals the device product of
the same operands and two random moduli."""
import threading

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# (an, bn, 64-bit digits)
SIZES = [(131072, 131073, True), (140000, 130001, True), (262144, 262144, True), (262145, 262144, True),
         (300007, 20011, True), (524288, 524288, True), (524289, 524288, True), (65537, 65537, False),
         (131072, 131072, False), (131073, 131072, False), (262144, 262144, False), (262144, 262145, False)]


def _device(gpu, torch, a, b):
    ta, tb = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    to = torch.empty(len(a) + len(b), dtype=torch.int64, device="cuda")
    gpu.mul_device(ta.data_ptr(), len(a), tb.data_ptr(), len(b), to.data_ptr())
    gpu.stream_check()
    return to.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("an,bn,wide", SIZES)
def test_overlapped_host_product(gpu, an, bn, wide):
    torch = pytest.importorskip("torch")
    prev = gpu.set_wide_digits(wide)
    try:
        a, b = O.splitmix64(an, an), O.splitmix64(bn + 1, bn)
        want = _device(gpu, torch, a, b)
        O.spot_check(want, a, b, an + bn)
        assert np.array_equal(gpu.mul(a, b), want)
        buf = np.zeros(an + bn, np.uint64)  # the result over operand a
        buf[:an] = a
        gpu.check(gpu.lib().prec_gpu_mul(gpu._p(buf), an, gpu._p(b), bn, gpu._p(buf)))
        assert np.array_equal(buf, want)
        s = gpu.sqr(a)
        O.spot_check(s, a, a, an)
    finally:
        gpu.set_wide_digits(prev)


def test_overlapped_two_threads(gpu):
    sizes = [(200000, 150000), (270000, 260000), (66000, 270000)]
    bad = []

    def run(seed):
        try:
            for i, (an, bn) in enumerate(sizes * 2):
                a, b = O.splitmix64(seed + i, an), O.splitmix64(seed + 50 + i, bn)
                O.spot_check(gpu.mul(a, b), a, b, seed + i)
        except Exception as e:  # noqa: BLE001 -- reported below
            bad.append(e)

    ts = [threading.Thread(target=run, args=(1000 * t,)) for t in (1, 2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
