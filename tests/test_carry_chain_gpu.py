"""GPU tests of carries between the blocks of the carry kernel: operands a and b
(one 32-bit word in its top limb) built so that the limb sums of a*b (low half of a_m b plus high half of
a_(m-1) b) are all ones over long runs, with and without a carry entering the
run, so that blocks cannot tell their carry-in from the limb below them.
Exact against Python's integers, by every path that runs the kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1
KINDS = ("long", "none", "runs")


def _chain(n, lb, kind):
    """(a, b): 'long' one carry through every limb, 'none' all ones and no carry,
    'runs' runs of all ones of up to three blocks, about half entered by a carry."""
    rng = np.random.default_rng(n)
    b = int(rng.integers(1 << 31, 1 << 32)) | 1
    inv = pow(b, -1, 1 << 64)
    rnd = rng.integers(1 << 63, 1 << 64, n, dtype=np.uint64).tolist()
    want = [M64] * n  # limb sum of position m; None: any
    if kind == "long":
        want[0], want[1] = None, 1 << 64
    elif kind == "runs":
        m = 0
        while m < n:
            want[m] = None
            if rng.random() < 0.5 and m + 1 < n:
                want[m + 1] = 1 << 64
            m += int(rng.integers(2, 3100))
    a, hi = [], 0
    for m in range(n):
        x = rnd[m] if want[m] is None else (want[m] - hi) * inv & M64
        a.append(x)
        hi = x * b >> 64
    return np.array(a, dtype=np.uint64), np.array([0] * (lb - 1) + [b], dtype=np.uint64)


def _exact(a, b):
    x = int.from_bytes(a.tobytes(), "little") * int(b[-1])
    return bytes(8 * (len(b) - 1)) + x.to_bytes(8 * (len(a) + 1), "little")


def _device(gpu, torch, a, b):
    ta, tb = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    to = torch.full((len(a) + len(b),), -1, dtype=torch.int64, device="cuda")
    gpu.mul_device(ta.data_ptr(), len(a), tb.data_ptr(), len(b), to.data_ptr())
    gpu.stream_check()
    return to.cpu().numpy().tobytes()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("n,lb", [(16400, 1), (65537, 1), (100000, 60000), (140001, 1), (250000, 60000),
                                  (500000, 100000), (900000, 300000)])
def test_carry_chain_single(gpu, n, lb, wide, kind):
    torch = pytest.importorskip("torch")
    prev = gpu.set_wide_digits(wide)
    try:
        a, b = _chain(n, lb, kind)
        want = _exact(a, b)
        assert _device(gpu, torch, a, b) == want
        assert gpu.mul(a, b, ntt=True).tobytes() == want
    finally:
        gpu.set_wide_digits(prev)


@pytest.mark.parametrize("persistent", [False, True])
def test_carry_chain_batch(gpu, monkeypatch, persistent):
    torch = pytest.importorskip("torch")
    if persistent:
        monkeypatch.setenv("PREC_GPU_BATCH_PERSISTENT", "1")
    ops = [_chain(n, lb, kind) for n, lb in ((3000, 1), (5000, 7), (12000, 1), (20000, 4000), (250000, 60000))
           for kind in KINDS]
    inp = torch.from_numpy(np.concatenate([np.concatenate(p) for p in ops]).view(np.int64)).cuda()
    out = torch.full_like(inp, -1)
    items, o = [], 0
    for a, b in ops:
        pa = inp.data_ptr() + 8 * o
        items.append((pa, len(a), pa + 8 * len(a), len(b), out.data_ptr() + 8 * o))
        o += len(a) + len(b)
    gpu.mul_batch(items, torch.cuda.current_stream().cuda_stream)
    res, o = out.cpu().numpy(), 0
    for a, b in ops:
        assert res[o:o + len(a) + len(b)].tobytes() == _exact(a, b), len(a)
        o += len(a) + len(b)
