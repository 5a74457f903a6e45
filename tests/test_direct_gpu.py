"""Direct (schoolbook) products of short operands, exact against integer
arithmetic at the edges of their digit blocks, thread groups and rules, with
random limbs and with all-ones limbs (carries through every limb)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = ("random", "ones", "high_zero")
# (longer, shorter): one block, one group, each class's limits and one past them
BATCH = [(1, 1), (3, 2), (4, 4), (5, 1), (31, 33), (63, 64), (64, 64), (65, 1), (65, 65), (127, 128), (128, 128),
         (129, 7), (200, 160), (256, 160), (256, 161), (257, 96), (511, 95), (512, 96), (512, 97), (513, 4)]
SINGLE = [(1, 1), (2, 1), (4, 3), (5, 5), (64, 60), (609, 608), (612, 1), (1024, 1000), (1217, 1216), (2048, 2048),
          (2049, 2047), (2433, 1700), (4096, 1024), (4096, 1025), (4095, 3), (4097, 16)]


def _limbs(rng, n, pattern):
    if pattern == "ones":
        return np.full(n, ~np.uint64(0), dtype=np.uint64)
    a = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if pattern == "high_zero":
        a[n - (n + 1) // 2:] = 0
    return a


def _exact(a, b):
    x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
    return np.frombuffer(x.to_bytes(8 * (len(a) + len(b)), "little"), dtype=np.uint64)


# with a product of the transform among them, and direct products alone (the
# kernels then read the caller's items, each class its own)
ONLY_DIRECT = [s for s in BATCH if s not in ((256, 161), (512, 97), (513, 4))]


@pytest.mark.parametrize("pattern", PATTERNS)
@pytest.mark.parametrize("only", (False, True))
def test_batch(gpu, pattern, only):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    kinds = ONLY_DIRECT if only else BATCH
    sizes = [s for s in kinds for _ in range(5)] + [(b, a) for a, b in kinds]
    ops = [(_limbs(rng, a, pattern), _limbs(rng, b, pattern)) for a, b in sizes]
    flat = torch.from_numpy(np.concatenate([x for p in ops for x in p]).view(np.int64)).cuda()
    out = torch.full_like(flat, -1)
    items, o = [], 0
    for a, b in sizes:
        items.append((flat.data_ptr() + 8 * o, a, flat.data_ptr() + 8 * (o + a), b, out.data_ptr() + 8 * o))
        o += a + b
    for oneshot in (True, False):
        out.fill_(-1)
        torch.cuda.synchronize()
        if oneshot:
            gpu.mul_batch(items)
        else:
            batch = gpu.Batch(items)
            batch.run()
            gpu.stream_check()
            batch.close()
        got, o = out.cpu().numpy().view(np.uint64), 0
        for (a, b), (x, y) in zip(sizes, ops):
            assert np.array_equal(got[o:o + a + b], _exact(x, y)), (oneshot, a, b)
            o += a + b


@pytest.mark.parametrize("pattern", PATTERNS)
def test_single(gpu, pattern):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    runs = []
    for i, (an, bn) in enumerate(SINGLE + [(b, a) for a, b in SINGLE] + [(n, n) for n in (1, 77, 1500)]):
        a, b = _limbs(rng, an, pattern), _limbs(rng, bn, pattern)
        ta = torch.from_numpy(a.view(np.int64)).cuda()
        tb = torch.from_numpy(b.view(np.int64)).cuda()
        # the output between two guards
        to = torch.full((an + bn + 2,), -7, dtype=torch.int64, device="cuda")
        runs.append((a, b, ta, tb, to))
    torch.cuda.synchronize()
    for i, (a, b, ta, tb, to) in enumerate(runs):  # streams in turn, all products in flight
        gpu.mul_device(ta.data_ptr(), len(a), tb.data_ptr(), len(b), to.data_ptr() + 8, streams[i % 3 % 2].cuda_stream)
    for s in streams:
        gpu.stream_check(s.cuda_stream)
    for a, b, _, _, to in runs:
        got = to.cpu().numpy().view(np.uint64)
        assert got[0] == got[-1] == np.uint64(-7 & (2**64 - 1))
        assert np.array_equal(got[1:-1], _exact(a, b)), (len(a), len(b))
