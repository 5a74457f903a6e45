"""Host-pointer products through the page-locked buffer (up to 32768 limbs in
all) and just past it: exact, from several threads, with zero high limbs,
with the result written over an operand, and with sizes falling and rising
on one thread."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 1), (193, 2), (300, 257), (6144, 6144), (6145, 3), (16384, 16384), (16385, 16384), (32767, 1),
         (32768, 1), (20000, 12768), (9, 32759), (9, 32760)]


def _exact(a, b):
    x = int.from_bytes(a.tobytes(), "little") * int.from_bytes(b.tobytes(), "little")
    return np.frombuffer(x.to_bytes(8 * (len(a) + len(b)), "little"), dtype=np.uint64)


def _check(gpu, seed):
    rng = np.random.default_rng(seed)
    for i in rng.permutation(len(SIZES)):
        an, bn = SIZES[i]
        a = rng.integers(0, 1 << 64, an, dtype=np.uint64)
        b = rng.integers(0, 1 << 64, bn, dtype=np.uint64)
        if i % 3 == 1:
            a[an - an // 3:] = 0
        want = _exact(a, b)
        assert np.array_equal(gpu.mul(a, b), want), (an, bn)
        buf = np.zeros(an + bn, np.uint64)  # the result over operand a
        buf[:an] = a
        gpu.check(gpu.lib().prec_gpu_mul(gpu._p(buf), an, gpu._p(b), bn, gpu._p(buf)))
        assert np.array_equal(buf, want), (an, bn)
        assert np.array_equal(gpu.sqr(a), _exact(a, a)), an


def test_sizes(gpu):
    _check(gpu, 5)


def test_threads(gpu):
    failed = []

    def one(seed):
        try:
            _check(gpu, seed)
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=one, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]
