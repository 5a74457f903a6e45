"""Transforms truncated to 5, 6 or 7 eighths: products whose coefficient count
lies at and just past each eighth of their transform length, on both digit
widths, as products, squares, uneven products and batches.  Exact against the
oracle up to 2^18 points; longer ones by the product modulo several primes."""
import numpy as np
import oracle as O
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = list(range(13, 19))


def _sizes(k, wide):
    """Limb pairs around e/8 of the 2^k-point transform."""
    per = 1 if wide else 2  # digits per limb
    out = []
    for e in (4, 5, 6, 7, 8):
        total = ((e << k) // 8 + 1) // per  # an + bn with an + bn - 1 (or 2(an+bn) - 1) coefficients at the edge
        for t in (total, total + 1):
            if per * t - 1 <= 1 << k:
                out += [(t // 2, t - t // 2), (t - t // 4, t // 4)]
        out.append((total // 2, 0))  # a square
    return out


def _operands(k, i, an, bn):
    a = O.splitmix64(1000 * k + i, an)
    if i % 4 == 3:
        a[:] = ~np.uint64(0)
    return a, (a if bn == 0 else O.splitmix64(1000 * k + i + 500, bn))


@pytest.mark.parametrize("k", LENGTHS)
def test_host_32bit(gpu, k):
    prev = gpu.set_wide_digits(False)
    try:
        for i, (an, bn) in enumerate(_sizes(k, False)):
            a, b = _operands(k, i, an, bn)
            assert np.array_equal(gpu.mul(a, b, ntt=True), O.mul_ntt(a, b)), (an, bn)
    finally:
        gpu.set_wide_digits(prev)


@pytest.mark.parametrize("k", (18, 20, 23))
def test_host_wide(gpu, k):
    for i, (an, bn) in enumerate(_sizes(k, True)):
        a, b = _operands(k, i, an, bn)
        got = gpu.mul(a, b, ntt=True)
        if k == 18:
            assert np.array_equal(got, O.mul_ntt(a, b)), (an, bn)
        else:
            O.spot_check(got, a, b, 7 * k + i)


def test_host_wide_long_rows(gpu):
    """2^22 points of 64-bit digits (2^10 columns, 2^12-point rows), and the same
    length once its table entry holds another configuration."""
    try:
        for i, (an, bn) in enumerate(_sizes(22, True)):
            a, b = _operands(22, i, an, bn)
            O.spot_check(gpu.mul(a, b, ntt=True), a, b, 22 + i)
        gpu.tune_set(**dict(gpu.tune_get(22), rows_per_cta=2))
        a, b = _operands(22, 0, 1500000, 1400001)
        O.spot_check(gpu.mul(a, b, ntt=True), a, b, 22)
    finally:
        gpu.tune_reset()


def test_long_32bit(gpu):
    """2^24 points of 32-bit digits: the reduced-residue set's kernels."""
    prev = gpu.set_wide_digits(False)
    try:
        for e in (5, 6, 7):
            t = (e << 24) // 16 - 3
            a, b = _operands(24, e, t // 2, t - t // 2)
            O.spot_check(gpu.mul(a, b, ntt=True), a, b, e)
    finally:
        gpu.set_wide_digits(prev)


def test_batch(gpu):
    """Every kept length of every class in one batch, enough of each that none
    is merged, and once more with single members (merged)."""
    torch = pytest.importorskip("torch")
    for copies in (40, 1):
        sizes = []
        for k in (13, 14, 16, 17):
            sizes += [(a, b) for a, b in _sizes(k, False) if b] * (copies if k < 17 else (copies + 3) // 4)
        sizes += [(a, b) for a, b in _sizes(18, True) if b]
        rng = np.random.default_rng(copies)
        flat = rng.integers(0, 1 << 64, sum(a + b for a, b in sizes), dtype=np.uint64)
        din = torch.from_numpy(flat.view(np.int64)).cuda()
        dout = torch.full_like(din, -1)
        items, o = [], 0
        for a, b in sizes:
            items.append((din.data_ptr() + 8 * o, a, din.data_ptr() + 8 * (o + a), b, dout.data_ptr() + 8 * o))
            o += a + b
        batch = gpu.Batch(items)
        batch.run()
        gpu.stream_check()
        batch.close()
        got, o = dout.cpu().numpy().view(np.uint64), 0
        for i, (a, b) in enumerate(sizes):
            if copies == 1 or i % 17 == 0:
                want = O.mul_ntt(flat[o:o + a], flat[o + a:o + a + b])
                assert np.array_equal(got[o:o + a + b], want), (a, b)
            o += a + b
