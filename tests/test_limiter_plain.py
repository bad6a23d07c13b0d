"""The FP64 limiters' bit-level and fast-reciprocal forms against the plain expressions
(tests/cpp/limiter_plain_check.cu), on the host and on the GPU: minmod and MC exactly, van Albada
and van Leer to their rounding, with zeros of both signs, subnormal, huge and infinite values and
NaN among the arguments."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("where", ["host", pytest.param("device", marks=pytest.mark.gpu)])
def test_limiters_against_the_plain_expressions(tmp_path, where):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "limiter_plain_check")
    # no contraction in the plain expressions on the host
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-gencode",
                    "arch=compute_103a,code=sm_103a", "--expt-relaxed-constexpr", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "limiter_plain_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe, where], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
