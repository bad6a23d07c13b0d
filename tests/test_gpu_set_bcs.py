"""A refused hc_set_bcs leaves a context as it was: the boundaries set before still hold, and the
next valid call gives the residual and the steps of a fresh context, whatever types the refused one
named."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300._capi import HCError
from hyperboliconvergence_gb300.solver import Mesh1D, Solver

pytestmark = pytest.mark.gpu


def run(s, q):
    s.set_state(q)
    r = s.residual()
    s.step(2)
    return r, s.get_state()


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("precision", ["fp64", "fp64_df", "fp32"])
@pytest.mark.parametrize("types", [["wall", "riemann", "periodic", "periodic"],
                                   ["periodic", "periodic", "fixed", "entropy"]])
def test_refused_boundaries_2d(precision, types):
    mesh, _, ref, q, sp = cases.quadrant_riemann(20, 35, np.random.default_rng(8))
    kw = dict(flux="roe", limiter="vanalbada", precision=precision, species=sp)
    periodic = ["periodic"] * 4
    s = Solver(mesh, periodic, None, **kw)
    before = run(s, q)
    with pytest.raises(HCError):
        s.set_bcs(types, None)
    assert same(run(s, q), before)
    partial = list(ref)
    partial[types.index("riemann") if "riemann" in types else 3] = None
    with pytest.raises(HCError):
        s.set_bcs(types, partial)
    s.set_bcs(types, ref)
    assert same(run(s, q), run(Solver(mesh, types, ref, **kw), q))
    # types that are refused as such
    with pytest.raises(HCError):
        s.set_bcs(["periodic", "wall", "wall", "wall"], ref)
    assert same(run(s, q), run(Solver(mesh, types, ref, **kw), q))


def test_refused_boundaries_1d():
    mesh, (left, right) = Mesh1D(np.linspace(0.0, 1.0, 41)), (np.array([0.1, 1.0, 1.0]), np.array([0.0, 0.125, 0.1]))
    x = mesh.centres()
    q = np.array([0.1 + 0 * x, 1.0 + 0.1 * np.sin(2 * np.pi * x), 1.0 + 0 * x])
    s = Solver(mesh, ["periodic", "periodic"], None, flux="roe", limiter="vanalbada")
    before = run(s, q)
    with pytest.raises(HCError):
        s.set_bcs(["riemann", "fixed"], [left, None])
    assert same(run(s, q), before)
    s.set_bcs(["riemann", "fixed"], [left, right])
    assert same(run(s, q), run(Solver(mesh, ["riemann", "fixed"], [left, right], flux="roe", limiter="vanalbada"), q))
