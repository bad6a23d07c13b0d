"""The host rules that pick the FP64 tile and the rows of an FP32 strip run
(tests/cpp/tile_rule_check.cu), over mesh sizes up to the launch limits; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_rules(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "tile_rule_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-o", exe, os.path.join(ROOT, "tests", "cpp", "tile_rule_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
