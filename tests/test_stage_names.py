"""The kernel names that the profile entry point reports are those of the kernels
the library has, in launch order (CPU)."""
import os
import re

from preclib_gb300 import build as B
from preclib_gb300 import native


def _names(path):
    out = []
    while True:
        n = native.lib().prec_gpu_stage_name(path, len(out)).decode()
        if not n:
            return out
        out.append(n)


def test_fp64_band_names_are_its_launches():
    src = open(os.path.join(B.CSRC, "fft_kernels.cu")).read()
    body = src[src.index("int fft_launch("):]
    order = []
    for n in re.findall(r"launch_pdl\(false, (k_\w+)|launch_carry<", body):
        order.append(n or "k_fft_carry")
    assert _names(2) == list(dict.fromkeys(order))


def test_ntt_names():
    assert _names(0) == ["k_small"]
    assert _names(1) == ["k_fwd_cols", "k_rows", "k_inv_cols", "k_crt_carry"]
    assert _names(3) == _names(-1) == []
