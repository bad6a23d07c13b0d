"""What the FP32 strip kernel leaves to the 8x32 tile -- the conserved basis -- with each limiter that
is a compile-time constant there, against the 4x32 tile, which chooses it at run time: the same
operations, up to how a product and a sum are contracted."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def conserved(q):
    return np.stack([q[2] * q[0], q[2] * q[1], q[2], q[3] / 0.4 + 0.5 * q[2] * (q[0] ** 2 + q[1] ** 2)])


@pytest.mark.parametrize("limiter", ["vanalbada", "vanleer", "minmod", "nolimit2", "nolimit3", "superbee"])
@pytest.mark.parametrize("flux,dt", [("roe", "local"), ("slau", "global")])
def test_conserved_tile(limiter, flux, dt):
    mesh, bc, ref, q, sp = cases.cylinder(21, 45, mach=0.4, rb=4.0)
    c = mesh.centres()
    q = conserved(q * (1 + 0.03 * np.sin(3 * c[0])[None] * np.cos(2 * c[1])[None]))
    ref = [None if r is None else conserved(r) for r in ref]
    out = []
    for tile in ("8x32", "4x32"):
        s = Solver(mesh, bc, ref, flux=flux, limiter=limiter, dt=dt, cfl=0.4, precision="fp32", species=sp,
                   basis="conserved", tile=tile)
        s.set_state(q)
        r = s.residual()
        s.step(2)
        out.append((r, s.get_state()))
    (ra, qa), (rb, qb) = out
    # a residual sums four face fluxes of the size p A; about a hundred operations of one rounding
    # each lie between the state and a flux
    scale = max(np.abs(q[3]).max(), 1.0) * np.hypot(*np.diff(mesh.nodes, axis=1).reshape(-1, 2).T).max()
    assert np.abs(ra - rb).max() <= 4 * 100 * 2.0 ** -24 * scale
    # and eight stages of CFL below 1 move a cell by less than that share of its faces' fluxes
    assert np.abs(qa - qb).max() <= 8 * 4 * 100 * 2.0 ** -24 * np.abs(q).max()
