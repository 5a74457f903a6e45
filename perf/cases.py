"""The measured work of this library: products of unsigned 64-bit limb
vectors through the public entry points of preclib_gb300.native.

listed()             the cases
draw(rng)            one more case of the same ranges
prepare(case, seed)  operands (uniform random limbs), plan or server
run(state)           one pass; its whole result as int64 limbs
exact(case, seed)    the same products without this library
work(case)           bytes a pass cannot do without

Kinds of case:
  host    prec_gpu_mul on pageable host vectors, the call that preclib's
          dispatcher makes (193 .. 6144 limbs: FP64 FFT band; above: NTT band)
  pinned  prec_gpu_mul on page-locked host vectors (the benchmark's end-to-end form)
  device  prec_gpu_mul_device on device vectors (the benchmark's kernel time
          and the Newton steps of the pi program)
  square  prec_gpu_mul_device with both operands the same vector (the
          squarings of the Newton steps)
  batch   a planned batch of uneven products, replayed (prec_gpu_batch_run)
  level   a one-shot batch (prec_gpu_mul_batch) of many short products: one
          level of a binary-splitting tree
  serve   a burst of requests of mixed sizes through the serving loop
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from preclib_gb300 import native, workloads


def listed():
    return [
        # the FFT band's short end: latency of one small host call
        {"name": "host_256x193", "kind": "host", "an": 256, "bn": 193},
        # the FFT band's benchmark product
        {"name": "host_3000x3000", "kind": "host", "an": 3000, "bn": 3000},
        # the NTT band's small benchmark product, as preclib calls it
        {"name": "host_8192x8192", "kind": "host", "an": 8192, "bn": 8192},
        # the headline product end to end (page-locked host memory)
        {"name": "pinned_1Mx1M", "kind": "pinned", "an": 1 << 20, "bn": 1 << 20},
        # the smallest device product of a Newton iteration (host arithmetic below 2^16 bits)
        {"name": "device_1024x1000", "kind": "device", "an": 1024, "bn": 1000},
        # a middle Newton step: ragged operands
        {"name": "device_20011x13001", "kind": "device", "an": 20011, "bn": 13001},
        # the headline product on the device
        {"name": "device_1Mx1M", "kind": "device", "an": 1 << 20, "bn": 1 << 20},
        # a squaring of a Newton step
        {"name": "square_300007", "kind": "square", "an": 300007, "bn": 300007},
        # the largest benchmark product
        {"name": "device_4Mx4M", "kind": "device", "an": 1 << 22, "bn": 1 << 22},
        # the batch benchmark: 4096 uneven products, 200 .. 65536 limbs
        {"name": "batch_4096", "kind": "batch", "count": 4096, "lo": 200, "hi": 65536, "sizes": 7},
        # the lowest device level of the pi program at 10^7 digits
        {"name": "level_44643", "kind": "level", "count": 44643, "lo": 58, "hi": 66, "sizes": 11},
        # a burst of requests, 256 .. 1048576 limbs, as the serving benchmark sends them
        {"name": "serve_64", "kind": "serve", "count": 64, "lo": 256, "hi": 1 << 20, "sizes": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pair(rng, lo, hi):
    n = _log_uniform(rng, lo, hi)
    m = max(1, int(n * rng.uniform(0.4, 1.0)))
    return (n, m) if rng.random() < 0.5 else (m, n)


def draw(rng):
    kind = rng.choice(["host", "host", "pinned", "device", "device", "device", "square", "batch", "level", "serve"])
    if kind in ("host", "pinned", "device"):
        an, bn = _pair(rng, *{"host": (193, 65536), "pinned": (6145, 1 << 20), "device": (1024, 1 << 22)}[kind])
        return {"kind": kind, "an": an, "bn": bn}
    if kind == "square":
        n = _log_uniform(rng, 1024, 1 << 22)
        return {"kind": kind, "an": n, "bn": n}
    seed = rng.randrange(1 << 20)
    if kind == "batch":
        return {"kind": kind, "count": _log_uniform(rng, 64, 4096), "lo": 200, "hi": _log_uniform(rng, 2000, 65536),
                "sizes": seed}
    if kind == "level":
        # from many products of a few tens of limbs (deep in the tree) to fewer, longer ones
        hi = _log_uniform(rng, 33, 1024)
        return {"kind": kind, "count": _log_uniform(rng, 500, 44643 * 66 // max(hi, 66)), "lo": hi - hi // 8, "hi": hi,
                "sizes": seed}
    return {"kind": kind, "count": _log_uniform(rng, 16, 64), "lo": 256, "hi": 1 << 20, "sizes": seed}


def _sizes(case):
    """(an, bn) of every product of a case."""
    kind = case["kind"]
    if kind in ("host", "pinned", "device", "square"):
        return [(case["an"], case["bn"])]
    rng = np.random.default_rng(case["sizes"])
    n = case["count"]
    if kind == "batch":
        lo, hi = workloads.batch_sizes(case["sizes"], n, case["lo"], case["hi"])
        return list(zip(hi.tolist(), lo.tolist()))
    if kind == "level":
        return list(zip(rng.integers(case["lo"], case["hi"] + 1, n).tolist(),
                        rng.integers(case["lo"], case["hi"] + 1, n).tolist()))
    s = np.rint(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), n))).astype(np.int64).tolist()
    return list(zip(s, s))


def work(case):
    limbs_in = limbs_out = 0
    for an, bn in _sizes(case):
        limbs_in += an if case["kind"] == "square" else an + bn
        limbs_out += an + bn
    return {"bytes": 8 * (limbs_in + limbs_out), "flops": 0}


def _random_device(seed, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, device="cuda", generator=g)
    x[n - 1] |= 1 << 40  # no zero top limb
    return x


def _operands(case, seed):
    """The operands of a single product, or every operand of a set end to end."""
    if case["kind"] in ("host", "pinned"):
        return (workloads.operand(2 * seed + 1, case["an"]), workloads.operand(2 * seed + 2, case["bn"]))
    if case["kind"] == "square":
        a = _random_device(seed, case["an"])
        return (a, a)
    if case["kind"] == "device":
        x = _random_device(seed, case["an"] + case["bn"])
        return (x[: case["an"]].clone(), x[case["an"]:].clone())
    return _random_device(seed, sum(an + bn for an, bn in _sizes(case)))


def prepare(case, seed):
    native.init(0)
    kind = case["kind"]
    if kind == "host":
        a, b = _operands(case, seed)
        return {"kind": kind, "a": a, "b": b}
    if kind == "pinned":
        a, b = (torch.from_numpy(x.view(np.int64)).pin_memory() for x in _operands(case, seed))
        out = torch.empty(a.numel() + b.numel(), dtype=torch.int64).pin_memory()
        u64p = ctypes.POINTER(ctypes.c_uint64)
        ptrs = [ctypes.cast(ctypes.c_void_p(t.data_ptr()), u64p) for t in (a, b, out)]
        return {"kind": kind, "a": a, "b": b, "out": out, "ptrs": ptrs}
    if kind in ("device", "square"):
        a, b = _operands(case, seed)
        out = torch.empty(a.numel() + b.numel(), dtype=torch.int64, device="cuda")
        return {"kind": kind, "a": a, "b": b, "out": out}
    data = _operands(case, seed)
    out = torch.empty_like(data)
    sizes = np.array(_sizes(case), dtype=np.int64)
    off = np.cumsum(sizes.sum(axis=1)) - sizes.sum(axis=1)
    items = np.empty((len(sizes), 5), dtype=np.uint64)  # prec_gpu_product_t: a, an, b, bn, out
    items[:, 0] = data.data_ptr() + 8 * off
    items[:, 1] = sizes[:, 0]
    items[:, 2] = data.data_ptr() + 8 * (off + sizes[:, 0])
    items[:, 3] = sizes[:, 1]
    items[:, 4] = out.data_ptr() + 8 * off
    state = {"kind": kind, "data": data, "out": out}
    if kind == "batch":
        state["plan"] = native.Batch([tuple(map(int, r)) for r in items])
    elif kind == "level":
        state["items"] = items
    else:
        state["requests"] = [tuple(map(int, r)) for r in items]
        state["server"] = native.Server(24 << 30, slots=16)
    return state


def run(state):
    kind = state["kind"]
    if kind == "host":
        return native.mul(state["a"], state["b"]).view(np.int64)
    if kind == "pinned":
        pa, pb, po = state["ptrs"]
        native.check(native.lib().prec_gpu_mul(pa, state["a"].numel(), pb, state["b"].numel(), po), "prec_gpu_mul")
        return state["out"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind in ("device", "square"):
        a, b, out = state["a"], state["b"], state["out"]
        native.mul_device(a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), out.data_ptr(), stream)
    elif kind == "batch":
        state["plan"].run(stream)
    elif kind == "level":
        items = state["items"]
        p = ctypes.cast(ctypes.c_void_p(items.ctypes.data), ctypes.POINTER(native.Product))
        native.check(native.lib().prec_gpu_mul_batch(p, len(items), stream or None), "prec_gpu_mul_batch")
    else:
        server = state["server"]
        for r in state["requests"]:
            server.submit(*r)
        server.drain()
    return state["out"]


def _product(a, b):
    """Exact product of two int64 limb vectors on the device: convolution of
    their bytes by a float64 FFT (sums below 2^42, error far below 1/2), then carries."""
    n = 8 * (a.numel() + b.numel())
    size = 1 << (n - 1).bit_length()
    fa = torch.fft.rfft(a.view(torch.uint8).to(torch.float64), n=size)
    fa *= torch.fft.rfft(b.view(torch.uint8).to(torch.float64), n=size)
    c = torch.round(torch.fft.irfft(fa, n=size)[:n]).to(torch.int64)
    while True:
        carry = c >> 8
        if not bool(carry.any()):
            break
        c &= 255
        c[1:] += carry[:-1]
    return c.to(torch.uint8).view(torch.int64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None  # minutes
    if kind in ("host", "pinned"):
        a, b = (torch.from_numpy(x.view(np.int64)).cuda() for x in _operands(case, seed))
        return _product(a, b).cpu()
    if kind in ("device", "square"):
        return _product(*_operands(case, seed))
    data = _operands(case, seed)
    out = torch.empty_like(data)
    if kind == "serve":
        o = 0
        for an, bn in _sizes(case):
            out[o: o + an + bn] = _product(data[o: o + an], data[o + an: o + an + bn])
            o += an + bn
        return out
    raw = data.cpu().numpy().tobytes()
    res = bytearray(len(raw))
    o = 0
    for an, bn in _sizes(case):
        m, e = o + 8 * an, o + 8 * (an + bn)
        x = int.from_bytes(raw[o:m], "little") * int.from_bytes(raw[m:e], "little")
        res[o:e] = x.to_bytes(e - o, "little")
        o = e
    return torch.from_numpy(np.frombuffer(res, dtype=np.int64).copy())
