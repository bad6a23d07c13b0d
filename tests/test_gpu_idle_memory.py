"""The device blocks that gradients keep for the next one: at most 2 GiB in a process whatever the
number of contexts, given back on request, and no reason for another context's allocation to fail."""
import gc

import numpy as np
import pytest
import torch

from hyperboliconvergence_gb300 import cases
from hyperboliconvergence_gb300.batch import Batch
from hyperboliconvergence_gb300.solver import Solver

pytestmark = pytest.mark.gpu
GB = 1 << 30


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def solver(n=512):
    mesh, bc, ref, q, sp = cases.cylinder(n, 2 * n)
    s = Solver(mesh, bc, ref, flux="roe", limiter="vanalbada", rk="ssp34", species=sp)
    s.set_state(q)
    return s


@pytest.fixture
def clean():
    gc.collect()
    torch.cuda.empty_cache()
    yield
    gc.collect()
    torch.cuda.empty_cache()


def gradients(solvers):
    # 16 stage tapes of 4 x 16.8 MB and some 0.5 GB of other blocks each
    return [s.gradient(15, snapshots=15, kind="drag")[:2] for s in solvers]


def release_idle():
    # looked up late, so that the bound is tested also where the call is missing
    import hyperboliconvergence_gb300
    hyperboliconvergence_gb300.release_idle()


def test_bound_over_contexts(clean):
    solvers = [solver() for _ in range(3)]
    for s in solvers:
        s.step(1)
    before = free()
    first = gradients(solvers)
    kept = before - free()
    assert 0.5 * GB < kept <= 2 * GB + 64 * (1 << 20)  # and the driver's own growth
    release_idle()
    assert before - free() <= 64 * (1 << 20)
    # the next gradients after a release are those of new contexts
    for s, fresh, (j, g) in zip(solvers, [solver() for _ in solvers], first):
        fresh.step(1)
        a, b = s.gradient(15, snapshots=15, kind="drag")[:2], fresh.gradient(15, snapshots=15, kind="drag")[:2]
        assert a[0] == b[0] and np.array_equal(a[1], b[1])


def test_idle_blocks_do_not_starve_others(clean):
    a = solver()
    a.step(1)
    before = free()
    gradients([a])
    assert before - free() > 0.5 * GB
    fill = torch.empty(free() - GB // 8, dtype=torch.uint8, device="cuda")
    try:
        b = solver()  # about 0.4 GB: only the idle blocks can make room for it
        b.step(2)
        rng = np.random.default_rng(2)
        batch = Batch([cases.gaussian_sum(64, 64, rng)[:4] for _ in range(8)], precision="fp64",
                      species=(1.4, 287.058, 0.3))
        batch.step_async(1)
        batch.sync()
    finally:
        del fill
        torch.cuda.empty_cache()
    a.step(1)
    b.step(0)
