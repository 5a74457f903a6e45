"""FP64 FFT band at the product lengths where the carry kernel's cluster is full
(4096, 8192 and 12288 limbs, one per thread more each): exact against integer
arithmetic, and the limbs past the product pass its check."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total", [n for t in (4096, 8192, 12288) for n in range(t - 3, t + 2) if n <= 12288])
def test_full_cluster(gpu, total):
    rng = np.random.default_rng(total)
    an = (total + 1) // 2
    bn = total - an
    for a, b in [(rng.integers(0, 1 << 64, an, dtype=np.uint64), rng.integers(0, 1 << 64, bn, dtype=np.uint64)),
                 (np.full(an, ~np.uint64(0)), np.full(bn, ~np.uint64(0)))]:
        x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
        assert gpu.mul(a, b, fft=True).tobytes() == x.to_bytes(8 * total, "little")
        assert gpu.last_stats().path == 2
