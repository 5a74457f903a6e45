"""GPU tests of the single-CTA transform (2^5 .. 2^12 points): the smallest and the
largest products of every length, alone between host arrays and in a batch,
whose short products run directly up to the edges named here; exact against
Python's integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(k):
    """(an, bn) whose 2 (an + bn) - 1 digits need 2^k points: fewest and most limbs."""
    lo, hi = (1 << (k - 2)) + 1, 1 << (k - 1)
    if k == 5:
        lo = 2
    out = []
    for total in {lo, lo + 1, hi - 1, hi}:
        out += [(total // 2, total - total // 2), (total - 1, 1), (total - total // 3, total // 3 or 1)]
    return [(a, b) for a, b in out if a > 0 and b > 0]


def _operands(rng, an, bn, kind):
    a = rng.integers(0, 1 << 64, an, dtype=np.uint64)
    b = rng.integers(0, 1 << 64, bn, dtype=np.uint64)
    if kind == "ones":
        a[:] = b[:] = ~np.uint64(0)
    elif kind == "sparse":
        a[:] = ~np.uint64(0)
        b[:] = 0
    a[-1] |= np.uint64(1 << 40)  # both top digits
    b[-1] |= np.uint64(1 << 40)
    return a, b


def _exact(a, b):
    x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
    return x.to_bytes(8 * (len(a) + len(b)), "little")


@pytest.mark.parametrize("k", range(5, 13))
def test_small_lengths_host(gpu, k):
    rng = np.random.default_rng(k)
    for an, bn in _edges(k):
        for kind in ("random", "ones", "sparse"):
            a, b = _operands(rng, an, bn, kind)
            assert gpu.mul(a, b, ntt=True).tobytes() == _exact(a, b), (an, bn, kind)
            st = gpu.last_stats()
            assert st.path == 0 and st.log2_n == k, (an, bn, st.log2_n)


def test_small_lengths_batch(gpu):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    sizes = [s for k in range(5, 13) for s in _edges(k)]
    # both sides of the direct product's edges
    sizes += [(192, 64), (192, 65), (191, 65), (200, 104), (200, 105), (256, 104), (105, 256), (257, 52), (53, 257),
              (459, 52), (460, 53), (461, 52), (416, 96), (97, 416), (512, 96), (512, 97)]
    ops = [_operands(rng, an, bn, ("random", "ones", "sparse")[i % 3]) for i, (an, bn) in enumerate(sizes)]
    inp = torch.from_numpy(np.concatenate([np.concatenate(p) for p in ops]).view(np.int64)).cuda()
    out = torch.full_like(inp, -1)
    items, o = [], 0
    for an, bn in sizes:
        pa, po = inp.data_ptr() + 8 * o, out.data_ptr() + 8 * o
        items.append((pa, an, pa + 8 * an, bn, po))
        o += an + bn
    gpu.mul_batch(items, torch.cuda.current_stream().cuda_stream)
    res, o = out.cpu().numpy(), 0
    for (an, bn), (a, b) in zip(sizes, ops):
        assert res[o:o + an + bn].tobytes() == _exact(a, b), (an, bn)
        o += an + bn
