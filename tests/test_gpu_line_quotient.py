"""The timestep of a short 1D line: cfl over the largest quotient of spectral radius and cell length,
each rounded once, in FP64 to the bit."""
import numpy as np
import pytest

from hyperboliconvergence_gb300.solver import Mesh1D, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [3, 31, 100, 257, 960])
def test_timestep_to_the_bit(nc):
    rng = np.random.default_rng(nc)
    for k in range(40):
        x = np.cumsum(np.concatenate([[0.0], rng.uniform(0.5, 1.5, nc) * 10.0 ** rng.uniform(-3, 3)]))
        q = np.stack([rng.uniform(-0.3, 0.3, nc), rng.uniform(0.8, 1.2, nc), rng.uniform(0.8, 1.2, nc)])
        s = Solver(Mesh1D(x), ["periodic"] * 2, None, flux="rusanov", limiter="vanalbada", rk="ssp11", cfl=0.4)
        s.set_state(q)
        lam = s.residual()[3]
        assert s.step(1).dt == 0.4 / (lam / np.diff(x)).max()
