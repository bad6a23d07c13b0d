"""The FP64 reciprocal, quotient, square roots, limiters and selections of the stage kernels
on the device (tests/cpp/fast_f64_check.cu): within the bounds of their derivation of the exact
values over the whole exponent range, and the plain expressions' results outside the fast
path's window (zero, subnormal, huge, infinite, NaN, negative)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_fast_f64_functions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fast_f64_check")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-o", exe, os.path.join(ROOT, "tests", "cpp", "fast_f64_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
