"""FP64 FFT band, every transform length 2^6 .. 2^16 (each has its own column
and row kernels) at its shortest and longest products, equal and uneven
operands, and limb patterns with long carry runs: exact against integer
arithmetic, the rounding distance far below 1/4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _limbs(rng, n, pattern):
    if pattern == "ones":
        return np.full(n, ~np.uint64(0), dtype=np.uint64)
    a = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if pattern == "sparse":  # runs of zero limbs below and between
        a[rng.random(n) < 0.95] = 0
        a[: n // 2] = 0
        a[-1] |= np.uint64(1)
    return a


@pytest.mark.parametrize("pattern", ("random", "ones", "sparse"))
def test_every_length(gpu, pattern):
    rng = np.random.default_rng(8)
    seen = set()
    n = 1
    sizes = []
    while n <= 6144:
        sizes += [(n, n), (n, max(1, n // 3)), (n, 1), (min(6144, n + 1), n)]
        n = n + 1 if n < 9 else int(n * 1.19) + 1
    sizes += [(6144, 6144), (6144, 6143), (6144, 2100)]
    for an, bn in sizes:
        a, b = _limbs(rng, an, pattern), _limbs(rng, bn, pattern)
        x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
        for u, v in ((a, b), (b, a)):
            got = gpu.mul(u, v, fft=True)
            assert got.tobytes() == x.to_bytes(8 * (an + bn), "little"), (an, bn)
            st = gpu.last_stats()
            assert st.path == 2 and st.fft_max_distance < 1e-3, (an, bn, st.fft_max_distance)
            seen.add(st.log2_n)
    assert seen == set(range(6, 17))
