"""The far fields' isentropic powers for gammas at and near the common gases' (tests/cpp/pow_gas_check.cu);
no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_powers_of_the_given_exponent(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    if __import__("platform").machine() != "x86_64":
        pytest.skip("long double is the reference")
    exe = str(tmp_path / "pow_gas_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "pow_gas_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
