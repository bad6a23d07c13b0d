"""The FP64 default tile, chosen by the mesh's size (8 x 8 and 4 x 8 cells on small meshes):
residuals, states and timesteps bit-identical to the 16 x 16 tile's on meshes smaller than,
equal to and ragged against each tile, for walls, far fields, periodic and fixed sides, and
through the adjoint's forward steps."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def case(kind, ni, nj):
    if kind == "cylinder":
        mesh, bc, ref, q, sp = cases.cylinder(ni, nj, mach=0.5, rb=6.0)
        c = mesh.centres()
        return mesh, bc, ref, q * (1 + 0.03 * np.sin(3 * c[0])[None] * np.cos(2 * c[1])[None]), sp
    return cases.quadrant_riemann(ni, nj, np.random.default_rng(ni * 100 + nj))


def run(c, tile, dt, limiter):
    mesh, bc, ref, q, sp = c
    s = Solver(mesh, bc, ref, flux="roe", limiter=limiter, dt=dt, species=sp)
    if tile:
        s.set_tile(tile)
    s.set_state(q)
    r = s.residual()
    st = s.step(3)
    return r, s.get_state(), st.dt


@pytest.mark.parametrize("kind,ni,nj", [("quadrant", 3, 3), ("quadrant", 4, 8), ("cylinder", 9, 17),
                                        ("cylinder", 40, 41), ("quadrant", 97, 131), ("cylinder", 8, 64),
                                        ("quadrant", 130, 121)])
@pytest.mark.parametrize("dt,limiter", [("local", "vanalbada"), ("global", "vanleer"), ("local", "minmod")])
def test_auto_tile_bit_identical(kind, ni, nj, dt, limiter):
    c = case(kind, ni, nj)
    a, b = run(c, None, dt, limiter), run(c, "16x16", dt, limiter)
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert a[2] == b[2]


def test_adjoint_of_a_small_mesh_independent_of_the_tile():
    mesh, bc, ref, q, sp = case("quadrant", 20, 27)
    out = []
    for tile in (None, "16x16"):
        s = Solver(mesh, bc, ref, flux="roe", limiter="vanalbada", species=sp)
        if tile:
            s.set_tile(tile)
        s.set_state(q)
        out.append(s.gradient(5, snapshots=2, kind="l2", target=q * 1.01)[:2])
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
