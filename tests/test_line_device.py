"""What the library keeps per device of a process, not only for the first one it ran on
(tests/cpp/line_device_check.cu, device_sms_check.cu): the short line's kernel made ready, the number
of SMs; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["line_device_check", "device_sms_check"])
def test_several_devices(tmp_path, name):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / name)
    # device code is not run: the quickest that nvcc makes of it will do
    subprocess.run([nvcc, "-std=c++17", "-O0", "-Xcicc", "-O0", "-gencode", "arch=compute_103a,code=compute_103a",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(ROOT, "tests", "cpp", name + ".cu")],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
