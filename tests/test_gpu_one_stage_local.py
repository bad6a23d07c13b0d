"""One-stage steps with local timesteps on meshes of several waves of blocks: the state after a step is
the conserved set plus the residual of the state before, nowhere of one that is already updated."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.batch import Batch
from hyperboliconvergence_gb300.solver import Mesh, Mesh1D, Solver

pytestmark = pytest.mark.gpu
G1 = 0.4
CFL = 0.7


def cons(q):
    if len(q) == 3:
        return np.stack([q[1] * q[0], q[1], q[2] / G1 + 0.5 * q[1] * q[0] ** 2])
    return np.stack([q[2] * q[0], q[2] * q[1], q[2], q[3] / G1 + 0.5 * q[2] * (q[0] ** 2 + q[1] ** 2)])


def prim(c):
    if len(c) == 3:
        return np.stack([c[0] / c[1], c[1], G1 * (c[2] - 0.5 * c[0] ** 2 / c[1])])
    return np.stack([c[0] / c[2], c[1] / c[2], c[2], G1 * (c[3] - 0.5 * (c[0] ** 2 + c[1] ** 2) / c[2])])


def advanced(q, res):
    return prim(cons(q) + res[:-1] * (CFL / res[-1]))


def box(ni, nj):
    x, y = (np.arange(ni) + 0.5) / ni, (np.arange(nj) + 0.5) / nj
    w = np.sin(6 * np.pi * x)[:, None] * np.cos(4 * np.pi * y)[None, :]
    # full steps on steep waves: a state that was read half updated is off by a share of w
    return Mesh.linspace(ni, nj, 0.0, 1.0, 0.0, 1.0), np.stack([0.5 + 0.2 * w, 0.2 - 0.2 * w, 1 + 0.3 * w, 1 + 0.2 * w])


def bound(precision):
    # some hundred roundings between a state and the next, residuals of order one times CFL
    return 300 * (2.0 ** -24 if precision == "fp32" else 2.0 ** -53 if precision == "fp64" else 2.0 ** -45)


@pytest.mark.parametrize("precision", ["fp64", "fp64_df", "fp32"])
@pytest.mark.parametrize("kw", [dict(flux="roe", limiter="vanalbada"), dict(flux="slau", limiter="superbee"),
                                dict(flux="rusanov", limiter="nolimit1", tile="4x32")])
def test_single_mesh(precision, kw):
    mesh, q = box(601, 1007)
    s = Solver(mesh, ["periodic"] * 4, None, rk="ssp11", dt="local", cfl=CFL, precision=precision, **kw)
    s.set_state(q)
    for _ in range(3):
        q = s.get_state()
        want = advanced(q, s.residual())
        s.step(1)
        assert np.abs(s.get_state() - want).max() <= bound(precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nc", [700, 20000])
def test_line(precision, nc):
    x = (np.arange(nc) + 0.5) / nc
    w = np.sin(2 * np.pi * 40 * x)
    q = np.stack([0.5 + 0.2 * w, 1 + 0.3 * w, 1 + 0.2 * w])
    s = Solver(Mesh1D(np.arange(nc + 1) / nc), ["periodic"] * 2, None, flux="roe", limiter="vanalbada", rk="ssp11",
               dt="local", cfl=CFL, precision=precision)
    s.set_state(q)
    for _ in range(3):
        q = s.get_state()
        want = advanced(q, s.residual())
        s.step(1)
        assert np.abs(s.get_state() - want).max() <= bound(precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["persistent", "per_instance", "graph"])
def test_batch(precision, mode):
    insts = [(m, ["periodic"] * 4, None, q) for m, q in (box(300, 411), box(640, 500), box(33, 900))]
    b = Batch(insts, flux="roe", limiter="vanalbada", rk="ssp11", dt="local", cfl=CFL, precision=precision)
    b.set_schedule("8x32", ctas_per_sm=1)
    if mode == "graph":
        b.capture(2)
        b.replay()
        b.replay()
    else:
        b.step_async(4, mode)
    b.sync()
    for k, (mesh, bc, _, q) in enumerate(insts):
        s = Solver(mesh, bc, None, flux="roe", limiter="vanalbada", rk="ssp11", dt="local", cfl=CFL,
                   precision=precision, species=(1.4, 287.058, 0.5))
        s.set_state(q)
        s.step(4)
        assert np.abs(b.get_state(k) - s.get_state()).max() <= 4 * bound(precision)


def test_scalar_law():
    mesh, bc, ref, q = cases.scalar_gaussian_sum(700, 900, np.random.default_rng(3))
    s = Solver(mesh, bc, ref, law="scalar", flux="rusanov", limiter="vanleer", rk="ssp11", dt="local", cfl=CFL)
    s.set_state(q)
    for _ in range(2):
        q = s.get_state()
        res = s.residual()
        s.step(1)
        assert np.abs(s.get_state() - (q + res[:-1] * (CFL / res[-1]))).max() <= bound("fp64")
