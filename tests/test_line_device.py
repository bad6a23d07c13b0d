"""The short line's kernel is made ready on every device that a process uses, not only on the first
(tests/cpp/line_device_check.cu); no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_line_kernel_on_several_devices(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "line_device_check")
    # device code is not run: the quickest that nvcc makes of it will do
    subprocess.run([nvcc, "-std=c++17", "-O0", "-Xcicc", "-O0", "-gencode", "arch=compute_103a,code=compute_103a",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(ROOT, "tests", "cpp", "line_device_check.cu")],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
