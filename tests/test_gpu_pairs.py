"""Packed pairs of double-float values (hc_pair.cuh): each operation rounds like the scalar one of
hc_df64.cuh, so both give the same bits; so does the split of a double by its bits.  Ties, carries
into the exponent, zeros, values outside FP32's range and non-finite ones are among the splits."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OPS = ("add", "sub", "mul", "div", "rcp", "vanalbada", "vanleer", "minmod", "state", "split", "split_wide", "roe")


@pytest.fixture(scope="module")
def mismatches(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pairs") / "pair_check")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(ROOT, "tests", "cpp", "pair_check.cu")],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {line.split()[0]: int(line.split()[1]) for line in out.splitlines()}


@pytest.mark.gpu
@pytest.mark.parametrize("op", OPS)
def test_packed_pairs_give_the_scalar_bits(mismatches, op):
    assert mismatches[op] == 0
