"""A call of no steps changes nothing: the state, the time, and the timestep and residual norm of the
last step, which its stats report."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.solver import Mesh1D, Solver

pytestmark = pytest.mark.gpu


def make(dim, precision, dt):
    if dim == 2:
        mesh, bc, ref, q, sp = cases.cylinder(24, 40)
        q = q * (1 + 0.02 * np.sin(3 * mesh.centres()[0]))
    else:
        mesh, bc, sp = Mesh1D(np.linspace(0.0, 1.0, 51)), ["riemann"] * 2, (1.4, 287.058, 1e-4)
        ref = [np.array([0.0, 1.0, 1.0]), np.array([0.0, 0.125, 0.1])]
        q = np.where(np.arange(50) < 25, ref[0][:, None], ref[1][:, None])
    s = Solver(mesh, bc, ref, flux="roe", limiter="vanalbada", precision=precision, dt=dt, species=sp)
    s.set_state(q)
    return s


@pytest.mark.parametrize("dim", [1, 2])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dt", ["global", "local"])
def test_no_steps(dim, precision, dt):
    s = make(dim, precision, dt)
    a = s.step(3)
    before, q = (a.dt, a.t, a.resnorm), s.get_state()
    assert a.resnorm > 0 and a.dt > 0
    b = s.step(0)
    assert (b.dt, b.t, b.resnorm) == before
    out = np.empty_like(q)
    c = s.step_host(q, out, 0)
    assert (c.dt, c.t, c.resnorm) == before
    assert np.array_equal(out, q) and np.array_equal(s.get_state(), q)
    # and the next steps are those of a context that was not asked for none
    f = make(dim, precision, dt)
    f.step(3)
    assert s.step(2).resnorm == pytest.approx(f.step(2).resnorm, rel=1e-12 if precision == "fp64" else 1e-5)
    assert np.array_equal(s.get_state(), f.get_state())
