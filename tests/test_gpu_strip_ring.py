"""The bounded wait of the FP32 strip kernel's record ring (tests/cpp/strip_ring_check.cu): the lanes
of a warp take one answer from it, in time or not."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_bounded_wait_is_one_answer_per_warp(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "strip_ring_check")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr",
                    "-o", exe, os.path.join(ROOT, "tests", "cpp", "strip_ring_check.cu")], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
