"""Short lines run in one cluster launch (up to 960 cells, 30-cell tiles, 64 steps a launch) and
longer ones by launches per stage: both against the 1D oracle, FP64, at sizes around a tile, a
block and the limit between the two, for every kind of end and both timestep modes; a run of
more steps than a launch takes equals the same steps one call at a time, bit for bit."""
import numpy as np
import pytest

from hyperboliconvergence_gb300.solver import Mesh1D, Solver
from oracle.oracle_py import OracleSolver1D

pytestmark = pytest.mark.gpu


def problem(nc, ends):
    rng = np.random.default_rng(nc)
    w = rng.uniform(0.8, 1.2, nc)
    if ends[0] == "periodic":
        w[:] = 1.0
    x = np.concatenate([[0.0], np.cumsum(w)]) / w.sum()
    c = 0.5 * (x[:-1] + x[1:])
    q = np.stack([0.3 + 0.1 * np.sin(2 * np.pi * c), 1 + 0.2 * np.cos(2 * np.pi * c), 0.8 + 0.1 * np.sin(4 * np.pi * c)])
    ref = [None if e in ("periodic", "wall") else np.array([0.3, 1.1, 0.75]) for e in ends]
    return x, q, ref


def solver(nc, ends, flux, limiter, dt, rk="ssp34", precision="fp64"):
    x, q, ref = problem(nc, ends)
    s = Solver(Mesh1D(x), list(ends), ref, flux=flux, limiter=limiter, rk=rk, dt=dt, cfl=0.5, precision=precision)
    s.set_state(q)
    return s


@pytest.mark.parametrize("nc", [3, 29, 30, 31, 61, 240, 241, 499, 960, 961])
@pytest.mark.parametrize("ends", [("periodic", "periodic"), ("wall", "riemann"), ("riemann", "entropy"), ("fixed", "wall")])
@pytest.mark.parametrize("flux,limiter,dt,rk", [("roe", "mc", "global", "ssp34"), ("slau", "vanalbada", "local", "ssp33")])
def test_line_matches_the_oracle(nc, ends, flux, limiter, dt, rk):
    x, q, ref = problem(nc, ends)
    s = solver(nc, ends, flux, limiter, dt, rk)
    o = OracleSolver1D(x, list(ends), flux=flux, limiter=limiter, rk=rk, dt=dt, cfl=0.5, ref=ref)
    o.set_state(q)
    s.step(3)
    o.step(3)
    a, b = s.get_state(), np.asarray(o.get_state()).reshape(3, nc)
    err = np.abs(a - b).max(axis=1) / np.abs(b).max(axis=1)
    assert err.max() <= 1e-12, err


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dt", ["global", "local"])
def test_chunks_of_steps_are_the_same_steps(precision, dt):
    a, b = (solver(128, ("riemann", "wall"), "roe", "mc", dt, precision=precision) for _ in range(2))
    sa = a.step(150)
    for _ in range(150):
        sb = b.step(1)
    assert np.array_equal(a.get_state(), b.get_state())
    assert sa.dt == sb.dt and sa.t == sb.t
    assert abs(sa.resnorm - sb.resnorm) <= 1e-6 * sb.resnorm  # the warps' sums in another order


def test_non_physical_state_is_reported():
    from hyperboliconvergence_gb300 import HCError
    s = solver(100, ("periodic", "periodic"), "roe", "mc", "global")
    _, q, _ = problem(100, ("periodic", "periodic"))
    q[2, 40] = -1.0
    s.set_state(q)
    with pytest.raises(HCError, match="non-physical"):
        s.step(2)
    _, q, _ = problem(100, ("periodic", "periodic"))
    s.set_state(q)
    s.step(2)
