"""A batch whose instance has more strips than the strip kernel's work list can hold (16 bits within
an instance), yet no more tiles than the tile kernel's: it runs, and equals the single mesh's FP32
steps to the FP32 kernels' rounding."""
import numpy as np
import pytest

from hyperboliconvergence_gb300.batch import Batch
from hyperboliconvergence_gb300.solver import Mesh, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [False, True])
def test_wide_instance(extra):
    ni, nj = 3, 1_900_000  # 59,375 tiles of 8 x 32 cells, 67,858 strips
    x = np.linspace(0.0, 3.0, ni + 1)[:, None]
    y = np.linspace(0.0, float(nj), nj + 1)[None, :]
    mesh = Mesh(np.stack(np.broadcast_arrays(x, y), axis=2))
    w = np.sin(2 * np.pi * np.arange(nj) / 50.0)[None, :] * np.ones((ni, 1))
    q = np.stack([0.3 + 0.1 * w, 0.2 - 0.1 * w, 1.0 + 0.1 * w, 1.0 + 0.05 * w])
    small = (Mesh.linspace(9, 11, 0.0, 1.0, 0.0, 1.0), ["periodic"] * 4, None, np.full((4, 9, 11), 1.0))
    insts = [(mesh, ["periodic"] * 4, None, q)] + ([small] if extra else [])
    kw = dict(flux="slau", limiter="vanalbada", rk="ssp22", precision="fp32", species=(1.4, 287.058, 0.5))
    b = Batch(insts, **kw)
    b.step_async(2)
    b.sync()
    s = Solver(mesh, ["periodic"] * 4, None, **kw)
    s.set_state(q)
    s.step(2)
    # two steps change the state by O(1); the two kernels' rounding differs by a few units of 2^-24
    # per stage, each scaled by at most the CFL number's share of a flux difference
    assert np.abs(b.get_state(0) - s.get_state()).max() <= 64 * 2.0 ** -24
    if extra:
        assert np.array_equal(b.get_state(1), small[3])
