"""The FP32 strip kernel (28-column strips marched row by row) against the 16 x 16 tile kernel,
an independent arrangement of the same arithmetic: residuals and states after three steps
agree to FP32 rounding (1e-5, as between tile shapes, of each variable's scale; a residual is a
sum of face fluxes that nearly cancel, so its rounding is that of the fluxes, whose scale is the
spectral radius times the conserved variable) on meshes of one strip, exactly filled, one column over, and of one run and several, with walls, far fields, fixed
and periodic sides."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def problem(kind, ni, nj):
    if kind in ("riemann", "entropy"):
        mesh, bc, ref, q, sp = cases.cylinder(ni, nj, mach=0.4, rb=6.0, far=kind)
        c = mesh.centres()
        return mesh, bc, ref, q * (1 + 0.03 * np.sin(3 * c[0])[None] * np.cos(2 * c[1])[None]), sp
    rng = np.random.default_rng(ni * 100 + nj)
    if kind == "fixed":
        return cases.quadrant_riemann(ni, nj, rng)
    mesh, bc, ref, q, sp = cases.gaussian_sum(ni, nj, rng)
    if kind == "walls":
        return mesh, ["wall"] * 4, None, q * np.array([0.1, 0.1, 1.0, 1.0])[:, None, None], sp
    return mesh, bc, ref, q, sp


def run(p, tile, flux, limiter, dt):
    mesh, bc, ref, q, sp = p
    s = Solver(mesh, bc, ref, flux=flux, limiter=limiter, dt=dt, precision="fp32", species=sp)
    if tile:
        s.set_tile(tile)
    s.set_state(q)
    r = s.residual()
    st = s.step(3)
    return r, s.get_state(), st


@pytest.mark.parametrize("ni,nj", [(3, 3), (4, 27), (5, 28), (9, 29), (33, 56), (17, 57), (64, 85)])
@pytest.mark.parametrize("kind", ["riemann", "entropy", "fixed", "periodic", "walls"])
@pytest.mark.parametrize("flux,limiter,dt", [("roe", "vanalbada", "local"), ("slau", "vanleer", "global"),
                                             ("ausmpup", "minmod", "local"), ("rusanov", "nolimit3", "global")])
def test_strips_match_tiles(kind, ni, nj, flux, limiter, dt):
    p = problem(kind, ni, nj)
    a, b = run(p, None, flux, limiter, dt), run(p, "16x16", flux, limiter, dt)
    q = p[3]
    e = q[3] / 0.4 + 0.5 * q[2] * (q[0] ** 2 + q[1] ** 2)
    m = np.sqrt(2 * q[2] * (e + q[3])).max()  # bounds rho (|u| + a)
    lam = b[0][4].max()
    flux = lam * np.array([m, m, q[2].max(), (e + q[3]).max(), 1.0])
    err = np.abs(a[0] - b[0]).reshape(5, -1).max(axis=1)
    assert (err <= 1e-5 * flux).all(), err / flux
    scale = np.abs(b[1]).reshape(4, -1).max(axis=1)
    scale[:2] = scale[:2].max()  # the two velocities together
    err = np.abs(a[1] - b[1]).reshape(4, -1).max(axis=1)
    assert (err <= 1e-5 * np.maximum(scale, scale.max() * 1e-3)).all(), err / scale
    assert abs(a[2].dt / b[2].dt - 1) <= 1e-5
    # the norm sums FP32 squares in another order
    assert abs(a[2].resnorm - b[2].resnorm) <= 1e-4 * b[2].resnorm
