"""A context set to a tile shape returns to the default choice, by the mesh's size in FP64: the
time of small steps is a new solver's again, the results never change."""
import time

import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300._capi import HC_ERR_ARG
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def seconds(s, q):
    s.set_state(q)
    s.step(20)
    best = 1e9
    for _ in range(5):
        t = time.perf_counter()
        s.step(100)
        best = min(best, time.perf_counter() - t)
    return best, s.get_state()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_back_to_the_default(precision):
    mesh, bc, ref, q, sp = cases.isentropic_vortex(40)
    s = Solver(mesh, bc, ref, flux="roe", limiter="vanleer", precision=precision, species=sp)
    new, a = seconds(s, q)
    s.set_tile("16x16/128")
    shape, _ = seconds(s, q)
    s.set_tile(None)
    back, b = seconds(s, q)
    assert s.tile is None
    assert np.array_equal(a, b)
    # 40 x 40 cells in nine 16 x 16 tiles take three times as long as the default's (FP64), twice (FP32)
    assert back < 1.25 * new and back < 0.8 * shape
    assert s.lib.hc_set_tile(s.h, -2) == HC_ERR_ARG and s.lib.hc_set_tile(s.h, 5) == HC_ERR_ARG
