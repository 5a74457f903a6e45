"""Truncated transforms, one product for each prime set, length and number of
eighths kept that has kernels of its own (template instantiations): 64-bit digits
at 2^19, 2^21, 2^24 and 2^25 points, 32-bit digits at 2^19 .. 2^26; and the batch
classes' wide column tiles of the lengths 2^15, 2^18 and 2^19.  By the product
modulo several primes."""
import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu


def _check(gpu, k, e, per, seed):
    total = ((e << k) // 8 + 1) // per  # the longest product of e eighths
    an = total // 2 + 3 * e
    a, b = O.splitmix64(seed, an), O.splitmix64(seed + 1, total - an)
    p = gpu.mul(a, b, ntt=True)
    st = gpu.last_stats()
    assert (st.log2_n, st.digit_bits) == (k, 64 // per)
    O.spot_check(p, a, b, seed)


@pytest.mark.parametrize("k,e", [(19, 5), (19, 6), (19, 7), (21, 5), (21, 6), (21, 7), (24, 5), (24, 6), (24, 7), (25, 5), (25, 6), (25, 7)])
def test_wide(gpu, k, e):
    _check(gpu, k, e, 1, 100 * k + e)


@pytest.mark.parametrize("k,e", [(k, e) for k in (19, 20, 21, 22, 23, 25, 26) for e in (5, 6, 7)])
def test_32bit(gpu, k, e):
    prev = gpu.set_wide_digits(False)
    try:
        _check(gpu, k, e, 2, 200 * k + e)
    finally:
        gpu.set_wide_digits(prev)


@pytest.mark.parametrize("k,per,copies", [(15, 2, 40), (18, 2, 3), (19, 1, 2)])
def test_batch(gpu, k, per, copies):
    """A class for each number of eighths that has kernels, with enough products
    that none is merged into another."""
    torch = pytest.importorskip("torch")
    sizes = []
    for e in (5, 6, 7, 8):
        total = ((e << k) // 8 + (e < 8)) // per
        long = min(total - total // 3, (1 << k) // 2 // per)  # both operands in the lower half
        sizes += [(total // 2, total - total // 2), (long, total - long)] * copies
    flat = np.random.default_rng(k).integers(0, 1 << 64, sum(a + b for a, b in sizes), dtype=np.uint64)
    din = torch.from_numpy(flat.view(np.int64)).cuda()
    dout = torch.full_like(din, -1)
    items, o = [], 0
    for a, b in sizes:
        assert gpu.ntt_log2(a, b) == k
        items.append((din.data_ptr() + 8 * o, a, din.data_ptr() + 8 * (o + a), b, dout.data_ptr() + 8 * o))
        o += a + b
    batch = gpu.Batch(items)
    # (at 2^15 points five eighths run with six and seven with all)
    assert batch.info()[0] == (2 if k == 15 else 4)
    batch.run()
    gpu.stream_check()
    batch.close()
    got, o = dout.cpu().numpy().view(np.uint64), 0
    for i, (a, b) in enumerate(sizes):
        if copies < 40 or i % 7 == 0:
            O.spot_check(got[o:o + a + b], flat[o:o + a], flat[o + a:o + a + b], i)
        o += a + b
