"""CPU checks of index arithmetic and small rules that kernels and launchers
share with the host: each program under host_checks/ includes the library's own
header, runs on the CPU and exits 0."""
import os
import subprocess

import pytest

from preclib_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DIR = os.path.join(ROOT, "tests", "host_checks")


def _check(name, tmp_path):
    exe = str(tmp_path / name)
    r = subprocess.run([B.nvcc(), *B.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-x", "cu", "-I", B.CSRC, "-o", exe,
                        os.path.join(DIR, name + ".cpp"), "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("name", sorted(f[:-4] for f in os.listdir(DIR) if f.endswith(".cpp")))
def test_host_check(name, tmp_path):
    _check(name, tmp_path)
