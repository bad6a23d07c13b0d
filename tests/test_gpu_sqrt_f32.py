"""The FP32 square root of the stage kernels on the device (tests/cpp/sqrt_f32_check.cu): within an ulp
over every exponent, and infinite, NaN, zero and negative arguments."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_fp32_square_root(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "sqrt_f32_check")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-o", exe, os.path.join(ROOT, "tests", "cpp", "sqrt_f32_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
