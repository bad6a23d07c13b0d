"""Gradients taken one after another from one context or batch (its blocks reused, its geometry
kept while the boundary types stay) equal those of fresh ones bit for bit: other step counts,
checkpoints and objectives in between, a dropped recording, new reference values and other
boundary types."""
import numpy as np
import pytest

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.batch import Batch
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu


def solver(ref, precision):
    mesh, bc, _, q, sp = cases.quadrant_riemann(21, 30, np.random.default_rng(4))
    s = Solver(mesh, bc, ref, flux="roe", limiter="vanalbada", precision=precision, species=sp)
    s.set_state(q)
    return s, q


def refs(scale=1.0):
    return [r * scale for r in cases.quadrant_riemann(21, 30, np.random.default_rng(4))[2]]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_context_reuse(precision):
    s, q = solver(refs(), precision)
    for nsteps, snaps, scale in [(6, 2, 1.0), (3, 0, 1.0), (9, 4, 1.01), (6, 2, 1.0)]:
        s.set_bcs(["fixed"] * 4, refs(scale))
        s.record(4, snapshots=3, kind="l2", target=q)  # dropped by the next one
        J, g, rb = s.gradient(nsteps, snapshots=snaps, kind="l2", target=1.01 * q)[:3]
        f, _ = solver(refs(scale), precision)
        J0, g0, rb0 = f.gradient(nsteps, snapshots=snaps, kind="l2", target=1.01 * q)[:3]
        assert J == J0 and np.array_equal(g, g0)
        assert all(np.array_equal(x, y) for x, y in zip(rb, rb0))
    # other boundary types rebuild the geometry
    s.set_bcs(["periodic"] * 4, None)
    mesh, _, _, _, sp = cases.quadrant_riemann(21, 30, np.random.default_rng(4))
    f = Solver(mesh, ["periodic"] * 4, None, flux="roe", limiter="vanalbada", precision=precision, species=sp)
    f.set_state(q)
    assert np.array_equal(s.residual(), f.residual())


def test_batch_reuse():
    rng = np.random.default_rng(9)
    insts = [cases.gaussian_sum(n, n + 5, rng)[:4] for n in (12, 30, 17)]
    targets = [1.02 * i[3] for i in insts]
    kw = dict(flux="rusanov", limiter="nolimit3", precision="fp32", species=(1.4, 287.058, 0.3))
    b = Batch(insts, **kw)
    for nsteps, snaps in [(5, 2), (8, 3), (2, 0), (5, 2)]:
        J, g, _ = b.gradient(nsteps, targets, snapshots=snaps)
        J0, g0, _ = Batch(insts, **kw).gradient(nsteps, targets, snapshots=snaps)
        assert np.array_equal(J, J0)
        assert all(np.array_equal(g[k], g0[k]) for k in g)
