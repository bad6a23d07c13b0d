"""The FP32 strip kernel's packed records take device memory only where they are used and where there
is room for them: not for configurations on the tile kernel, and not where they would take more than
a quarter of the free memory (a long narrow mesh), which then runs on the tile kernel."""
import gc

import numpy as np
import pytest
import torch

from hyperboliconvergence_gb300.batch import Batch
from hyperboliconvergence_gb300.solver import Mesh, Solver

pytestmark = pytest.mark.gpu
MB = 1 << 20


def records(ni, nj):
    return (nj + 27) // 28 * (ni + 3) * 27 * 32 * 4


def taken(make):
    gc.collect()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    keep = make()
    used = free - torch.cuda.mem_get_info()[0]
    del keep
    return used


def state(ni, nj):
    w = np.sin(2 * np.pi * np.arange(ni) / ni)[:, None] * np.ones((1, nj))
    return np.stack([0.3 + 0.1 * w, 0.2 - 0.1 * w, 1.0 + 0.1 * w, 1.0 + 0.05 * w])


@pytest.mark.parametrize("kw", [dict(limiter="superbee"), dict(limiter="vanalbada", basis="conserved")])
def test_no_records_without_strips(kw):
    ni, nj = 700, 1100
    mesh, q = Mesh.linspace(ni, nj, 0.0, 1.0, 0.0, 1.0), state(ni, nj)

    def single(**k):
        s = Solver(mesh, ["periodic"] * 4, None, flux="slau", precision="fp32", **k)
        s.set_state(q)
        return s

    def batch(**k):
        return Batch([(mesh, ["periodic"] * 4, None, q)], flux="slau", precision="fp32", **k)

    for make in (single, batch):
        make(**kw)  # the first use of a configuration loads its kernels
        make(limiter="vanalbada")
        with_strips, without = taken(lambda: make(limiter="vanalbada")), taken(lambda: make(**kw))
        # allocations are rounded to 2 MB at most
        assert with_strips - without >= records(ni, nj) - 4 * MB


def test_narrow_mesh_keeps_its_room():
    ni, nj = 400_000, 3
    x, y = np.linspace(0.0, float(ni), ni + 1)[:, None], np.linspace(0.0, 3.0, nj + 1)[None, :]
    mesh, q = Mesh(np.stack(np.broadcast_arrays(x, y), axis=2)), state(ni, nj)
    kw = dict(flux="slau", limiter="vanalbada", rk="ssp22", precision="fp32", dt="local")

    def make():
        s = Solver(mesh, ["periodic"] * 4, None, **kw)
        s.set_state(q)
        s.step(2)
        return s

    roomy = make().get_state()
    gc.collect()
    torch.cuda.empty_cache()
    assert records(ni, nj) > 5 * 1024 * MB // 4
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 5 * 1024 * MB, dtype=torch.uint8, device="cuda")
    tight = []
    try:
        used = taken(lambda: tight.append(make().get_state()) or make())
    finally:
        del fill
        torch.cuda.empty_cache()
    assert used < records(ni, nj)
    # the two kernels differ by the rounding of FP32
    assert np.abs(tight[0] - roomy).max() <= 64 * 2.0 ** -24
