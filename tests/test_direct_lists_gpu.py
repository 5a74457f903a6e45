"""Batches of direct products alone (the kernels read the caller's items, each
class by its index list made on the device) at the limits of every class of the
rule, one class alone (no list), more products of a class than one grid takes
(every group loops), and a batch one limb past each limit (the transform's).
Exact against integer arithmetic; the route by the number of launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (longer, shorter) limbs at each class's limits
CLASSES = [[(1, 1), (3, 2), (4, 4), (33, 31), (64, 1), (64, 64)],
           [(65, 1), (65, 65), (95, 12), (96, 96)],
           [(97, 1), (97, 96), (127, 113), (128, 128)],
           [(129, 1), (129, 64), (192, 64), (193, 104), (256, 104)],
           [(257, 1), (257, 52), (460, 52), (461, 96), (512, 96)]]
PAST = [(129, 65), (193, 105), (256, 105), (257, 53), (461, 97), (512, 97), (513, 4)]


def _limbs(rng, n, pattern):
    return np.full(n, ~np.uint64(0), dtype=np.uint64) if pattern == "ones" else rng.integers(0, 1 << 64, n, dtype=np.uint64)


def _check(gpu, sizes, pattern, launches):
    torch = pytest.importorskip("torch")
    flat = _limbs(np.random.default_rng(5), sum(a + b for a, b in sizes), pattern)
    din = torch.from_numpy(flat.view(np.int64)).cuda()
    out = torch.empty_like(din)
    items, want, o = [], bytearray(), 0
    for a, b in sizes:
        items.append((din.data_ptr() + 8 * o, a, din.data_ptr() + 8 * (o + a), b, out.data_ptr() + 8 * o))
        x, y = (int.from_bytes(flat[i:j].tobytes(), "little") for i, j in ((o, o + a), (o + a, o + a + b)))
        want += (x * y).to_bytes(8 * (a + b), "little")
        o += a + b
    batch = gpu.Batch(items)
    for run in ("one-shot", "first", "replay"):
        out.fill_(-1)
        torch.cuda.synchronize()
        before = gpu.launch_count()
        if run == "one-shot":
            gpu.mul_batch(items)
        else:
            batch.run()
            gpu.stream_check()
        assert launches is None or gpu.launch_count() - before == launches, run
        got = out.cpu().numpy().tobytes()
        assert got == bytes(want), (run, next(i for i in range(0, len(got), 8) if got[i:i + 8] != want[i:i + 8]) // 8)
    batch.close()


@pytest.mark.parametrize("pattern", ("random", "ones"))
def test_every_class(gpu, pattern):
    sizes = [s for c in CLASSES for s in c for _ in range(7)] + [(b, a) for c in CLASSES for a, b in c]
    _check(gpu, sizes, pattern, len(CLASSES) + 1)


@pytest.mark.parametrize("cls", range(len(CLASSES)))
def test_one_class(gpu, cls):
    _check(gpu, CLASSES[cls] * 3, "random", 1)


def test_more_than_a_grid(gpu):
    """64 CTAs per SM: 8 products each in the first two classes, 4 in the
    third, one in the last two."""
    import torch
    ctas = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [(2, 1)] * (8 * ctas + 100) + [(65, 1)] * 9 + [(97, 1)] * 9 + [(129, 1)] * (ctas + 50) + [(257, 1)] * (ctas + 3)
    order = np.random.default_rng(6).permutation(len(sizes))
    _check(gpu, [sizes[i] for i in order], "random", len(CLASSES) + 1)


def test_one_past(gpu):
    _check(gpu, [s for c in CLASSES for s in c] + PAST * 2 + [(b, a) for a, b in PAST], "random", None)
