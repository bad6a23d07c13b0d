"""Performance cases: the work a user of this framework has it do, through its public Python
entry points, over the range of sizes, precisions and options it is used in.

Families (the key "kind" of a case):
  tube      Solver on a Mesh1D: the reference's shock-tube driver (Sod, Roe + MC, ssp34, CFL 0.8)
  single    Solver on a 2D mesh: device state in, a few RK steps, device state out
  hosted    Solver.step_host: a host-resident field advanced in one call (integrate() as the
            reference's callers see it), copies included
  batch     Batch: an ensemble of uneven meshes, captured once as a CUDA graph and replayed
  adjoint   autograd.run_objective and its backward: drag of a cylinder run
  badjoint  autograd.batch_l2_objective and its backward: L2 losses of an ensemble

`exact` restates the path in plain torch float64 (least-squares gradients, MUSCL, fluxes,
boundaries, the RK tables); the gradients come from torch's own autograd through it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

GAMMA, R_AIR = 1.4, 287.058


# ------------------------------------------------------------------------- the cases
def listed():
    return [
        # smallest calls: the reference's shock-tube driver, 128 cells; launches and latency count
        {"name": "tube_128_fp64", "kind": "tube", "nc": 128, "flux": "roe", "limiter": "mc", "rk": "ssp34",
         "precision": "fp64", "steps": 20},
        # the small plain configuration: isentropic vortex, 128 x 128 periodic, global timestep
        {"name": "vortex_128_fp64", "kind": "single", "mesh": "vortex", "ni": 128, "nj": 128, "mach": 0.0,
         "flux": "roe", "limiter": "vanleer", "rk": "ssp34", "dt": "global", "precision": "fp64", "steps": 10},
        # a small ragged FP32 mesh: one member of an ensemble run by itself
        {"name": "quadrants_97x131_fp32", "kind": "single", "mesh": "quadrants", "ni": 97, "nj": 131, "mach": 0.0,
         "flux": "slau", "limiter": "vanalbada", "rk": "ssp34", "dt": "global", "precision": "fp32", "steps": 10},
        # the large plain configuration (the benchmark's headline), in each precision
        {"name": "cylinder_512x1024_fp64", "kind": "single", "mesh": "cylinder", "ni": 512, "nj": 1024, "mach": 0.3,
         "flux": "roe", "limiter": "vanalbada", "rk": "ssp34", "dt": "local", "precision": "fp64", "steps": 2},
        {"name": "cylinder_512x1024_fp32", "kind": "single", "mesh": "cylinder", "ni": 512, "nj": 1024, "mach": 0.3,
         "flux": "roe", "limiter": "vanalbada", "rk": "ssp34", "dt": "local", "precision": "fp32", "steps": 10},
        {"name": "cylinder_512x1024_df64", "kind": "single", "mesh": "cylinder", "ni": 512, "nj": 1024, "mach": 0.3,
         "flux": "roe", "limiter": "vanalbada", "rk": "ssp34", "dt": "local", "precision": "fp64_df", "steps": 2},
        # the same flow at Mach 0.8 with AUSM+up on a mesh whose sizes are no multiple of anything
        {"name": "cylinder_301x715_fp32", "kind": "single", "mesh": "cylinder", "ni": 301, "nj": 715, "mach": 0.8,
         "flux": "ausmpup", "limiter": "vanleer", "rk": "ssp34", "dt": "local", "precision": "fp32", "steps": 10},
        # a host field advanced end to end, copies included
        {"name": "quadrants_300x401_host", "kind": "hosted", "mesh": "quadrants", "ni": 300, "nj": 401, "mach": 0.0,
         "flux": "slau", "limiter": "vanalbada", "rk": "ssp34", "dt": "global", "precision": "fp64", "steps": 2},
        # the ensemble: uneven quadrant problems in one CUDA graph; larger and smaller members
        {"name": "batch_24_uneven_fp32", "kind": "batch", "n": 24, "lo": 64, "hi": 512, "of": 32, "flux": "slau",
         "limiter": "vanalbada", "rk": "ssp34", "precision": "fp32", "steps": 20},
        {"name": "batch_96_small_fp32", "kind": "batch", "n": 96, "lo": 16, "hi": 128, "of": 1, "flux": "slau",
         "limiter": "vanalbada", "rk": "ssp34", "precision": "fp32", "steps": 6},
        # gradient of the time-averaged drag with respect to the initial state and the far field
        {"name": "adjoint_256x512_fp64", "kind": "adjoint", "ni": 256, "nj": 512, "mach": 0.4, "flux": "roe",
         "limiter": "vanalbada", "rk": "ssp34", "precision": "fp64", "steps": 8, "snapshots": 3},
        # gradients of the L2 losses of an ensemble, one batched adjoint
        {"name": "batch_adjoint_8_fp32", "kind": "badjoint", "n": 8, "lo": 128, "hi": 512, "of": 64,
         "flux": "rusanov", "limiter": "nolimit3", "rk": "ssp34", "precision": "fp32", "steps": 8, "snapshots": 3},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "single", "single", "single", "single", "hosted", "batch", "adjoint", "badjoint"])
    rk = rng.choice(["ssp34", "ssp34", "ssp33", "ssp22"])
    if kind == "tube":
        return {"kind": kind, "nc": _size(rng, 48, 20000), "flux": rng.choice(["roe", "slau", "ausmpup"]),
                "limiter": rng.choice(["mc", "vanalbada", "minmod"]), "rk": rk,
                "precision": rng.choice(["fp64", "fp32"]), "steps": rng.randint(5, 20)}
    limiter = rng.choice(["vanalbada", "vanleer", "minmod"])
    if kind in ("single", "hosted"):
        mesh = rng.choice(["cylinder", "quadrants", "vortex"])
        prec = "fp64" if kind == "hosted" else rng.choice(["fp64", "fp32", "fp32", "fp64_df"])
        ni, nj = _size(rng, 40, 512), _size(rng, 40, 1024)
        if mesh == "vortex":
            nj = ni
        return {"kind": kind, "mesh": mesh, "ni": ni, "nj": nj,
                "mach": round(rng.uniform(0.3, 0.8), 3) if mesh == "cylinder" else 0.0,
                "flux": rng.choice(["roe", "slau", "ausmpup"]), "limiter": limiter, "rk": rk,
                "dt": rng.choice(["local", "global"]), "precision": prec,
                "steps": rng.randint(3, 10) if prec == "fp32" else rng.randint(1, 2)}
    if kind == "batch":
        small = rng.random() < 0.5
        return {"kind": kind, "n": rng.randint(16, 64) if small else rng.randint(8, 20), "lo": 16 if small else 64,
                "hi": 128 if small else 512, "of": rng.choice([1, 4, 32]) if small else rng.choice([4, 32]),
                "flux": rng.choice(["slau", "roe"]), "limiter": limiter, "rk": rk, "precision": "fp32",
                "steps": rng.randint(2, 6)}
    if kind == "adjoint":
        return {"kind": kind, "ni": _size(rng, 40, 256), "nj": _size(rng, 64, 512),
                "mach": round(rng.uniform(0.3, 0.5), 3), "flux": rng.choice(["roe", "rusanov"]),
                "limiter": rng.choice(["vanalbada", "nolimit3"]), "rk": rk, "precision": "fp64",
                "steps": rng.randint(3, 8), "snapshots": rng.randint(1, 4)}
    return {"kind": kind, "n": rng.randint(2, 8), "lo": 64, "hi": 320, "of": rng.choice([1, 32]), "flux": "rusanov",
            "limiter": "nolimit3", "rk": rk, "precision": "fp32", "steps": rng.randint(3, 8),
            "snapshots": rng.randint(1, 4)}


# ------------------------------------------------------------------------- inputs
def _cylinder_nodes(nr, nth, rc=0.5, rb=20.0, s=1.01):
    """O-grid of nr radial x nth circumferential cells, geometric radial stretching."""
    i = np.arange(nr + 1)
    r = rc + (rb - rc) * (s - 1.0) / (s ** nr - 1.0) * (s ** i - 1.0) / (s - 1.0)
    th = np.arange(nth + 1) * (2.0 * math.pi / nth)
    return np.stack([r[:, None] * np.cos(th), r[:, None] * np.sin(th)], axis=2)


def _box_nodes(ni, nj, length):
    x, y = np.arange(ni + 1) * (length / ni), np.arange(nj + 1) * (length / nj)
    return np.stack(np.broadcast_arrays(x[:, None], y[None, :]), axis=2).copy()


def _waves(rng, ni, nj, eps):
    """1 + a smooth field of size eps, periodic in j: four seeded modes per variable."""
    a = np.arange(ni)[:, None] / ni
    b = np.arange(nj)[None, :] / nj
    out = np.ones((4, ni, nj))
    for v in range(4):
        for _ in range(4):
            ki, kj = rng.integers(1, 5, 2)
            p, r = rng.uniform(0, 2 * math.pi, 2)
            out[v] += 0.25 * eps * rng.uniform(0.3, 1.0) * np.sin(math.pi * ki * a + p) * np.sin(
                2 * math.pi * int(kj) * b + r)
    return out


def _quadrants(rng, ni, nj):
    """Four-quadrant Riemann data: rho in [0.5, 2], p in [0.1, 2], |u|, |v| <= 1; draws whose
    interfaces separate faster than a fifth of the vacuum speed are drawn again."""
    while True:
        s = np.empty((4, 4))
        s[:, 2], s[:, 3] = rng.uniform(0.5, 2.0, 4), rng.uniform(0.1, 2.0, 4)
        s[:, :2] = rng.uniform(-1.0, 1.0, (4, 2))
        a = np.sqrt(GAMMA * s[:, 3] / s[:, 2])
        if all(s[h, c] - s[l, c] < 0.4 / (GAMMA - 1.0) * (a[l] + a[h])
               for l, h, c in ((0, 2, 0), (1, 3, 0), (0, 1, 1), (2, 3, 1))):
            break
    x = (np.arange(ni) + 0.5) / ni >= 0.5
    y = (np.arange(nj) + 0.5) / nj >= 0.5
    return np.moveaxis(s[2 * x[:, None].astype(int) + y[None, :]], 2, 0).copy()


def _mesh_inputs(case, rng):
    """nodes, boundary types, reference layers, primitive state, minf of one 2D problem."""
    ni, nj, kind = case["ni"], case["nj"], case["mesh"]
    if kind == "cylinder":
        qinf = np.array([case["mach"], 0.0, 1.0, 1.0 / GAMMA])
        # the freestream with a smooth disturbance (the second velocity's scaled by the first)
        w = _waves(rng, ni, nj, 0.05)
        q = qinf[:, None, None] * w
        q[1] = case["mach"] * (w[1] - 1.0)
        far = case.get("far", "riemann")
        return (_cylinder_nodes(ni, nj), ["wall", far, "periodic", "periodic"],
                [None, np.repeat(qinf[:, None], nj, axis=1), None, None], q, case["mach"])
    if kind == "vortex":
        c = (np.arange(ni) + 0.5) * (10.0 / ni)
        x0, y0 = rng.uniform(3.0, 7.0, 2)
        beta = rng.uniform(4.0, 5.0)
        dx = ((c - x0 + 5.0) % 10.0 - 5.0)[:, None]
        dy = ((c - y0 + 5.0) % 10.0 - 5.0)[None, :]
        r2 = dx * dx + dy * dy
        e = beta / (2 * math.pi) * np.exp(0.5 * (1.0 - r2))
        temp = 1.0 - (GAMMA - 1.0) * beta ** 2 / (8.0 * GAMMA * math.pi ** 2) * np.exp(1.0 - r2)
        rho = temp ** (1.0 / (GAMMA - 1.0))
        return (_box_nodes(ni, nj, 10.0), ["periodic"] * 4, None,
                np.stack([1.0 - dy * e, 1.0 + dx * e, rho, rho ** GAMMA]), math.sqrt(2.0 / GAMMA))
    q = _quadrants(rng, ni, nj)
    return (_box_nodes(ni, nj, 1.0), ["fixed"] * 4, [q[:, 0], q[:, -1], q[:, :, 0], q[:, :, -1]], q, 0.5)


def _tube_inputs(case, rng):
    """Sod's tube with seeded sides near (1, 1) and (0.125, 0.1): nodes, ends' values, {u, rho, p}."""
    nc = case["nc"]
    left = np.array([0.0, rng.uniform(0.9, 1.1), rng.uniform(0.9, 1.1)])
    right = np.array([0.0, rng.uniform(0.11, 0.14), rng.uniform(0.09, 0.11)])
    x = np.arange(nc + 1) * (1.0 / nc)
    q = np.where((0.5 * (x[:-1] + x[1:]) < 0.5)[None, :], left[:, None], right[:, None])
    return x, [left, right], q


def _members(case, rng):
    """The members of an ensemble: (nodes, bc, ref, state) of quadrant problems, or of Gaussian
    sums on the periodic unit square with their targets."""
    lo, hi, of = case["lo"], case["hi"], case["of"]
    # sizes from the range alone, so that every seed's ensemble is the same amount of work
    sizes = np.random.default_rng(lo * 7919 + hi * 31 + case["n"])
    out = []
    for _ in range(case["n"]):
        ni, nj = (int(v) * of for v in sizes.integers(-(-lo // of), hi // of + 1, 2))
        if case["kind"] == "batch":
            q = _quadrants(rng, ni, nj)
            out.append((_box_nodes(ni, nj, 1.0), ["fixed"] * 4, [q[:, 0], q[:, -1], q[:, :, 0], q[:, :, -1]], q, None))
        else:
            q, t = (_gaussians(rng, ni, ni) for _ in range(2))
            out.append((_box_nodes(ni, ni, 1.0), ["periodic"] * 4, None, q, t))
    return out


def _gaussians(rng, ni, nj):
    x, y = ((np.arange(ni) + 0.5) / ni)[:, None], ((np.arange(nj) + 0.5) / nj)[None, :]
    q = np.empty((4, ni, nj))
    q[0], q[1], q[2], q[3] = 0.5, 0.25, 5.0, 1.0
    for _ in range(8):
        cx, cy, w, amp = rng.uniform(0, 1), rng.uniform(0, 1), rng.uniform(0.02, 0.2), rng.uniform(-0.5, 0.5)
        q[2] += amp * np.exp(-(x - cx) ** 2 / (2 * w * w)) * np.exp(-(y - cy) ** 2 / (2 * w * w))
    return q


def _adjoint_inputs(case, rng):
    return _mesh_inputs(dict(case, mesh="cylinder", far="fixed"), rng)


# drag coefficient of the unit-diameter body at the freestream's dynamic pressure
def _cd_scale(mach):
    return 1.0 / (0.5 * mach * mach)


# ------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    from hyperboliconvergence_gb300.batch import Batch
    from hyperboliconvergence_gb300.solver import Mesh, Mesh1D, Solver
    rng = np.random.default_rng(seed)
    kind, opts = case["kind"], {k: case[k] for k in ("flux", "limiter", "rk", "precision")}
    real = torch.float32 if case["precision"] == "fp32" else torch.float64
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "tube":
        x, ref, q = _tube_inputs(case, rng)
        s = Solver(Mesh1D(x), ["riemann", "riemann"], ref, dt="global", cfl=0.8, stream=stream, **opts)
        q0 = torch.tensor(q, dtype=real, device="cuda")
        return {"case": case, "solver": s, "q0": q0, "out": torch.empty_like(q0)}
    if kind in ("single", "hosted"):
        nodes, bc, ref, q, minf = _mesh_inputs(case, rng)
        s = Solver(Mesh(nodes), bc, ref, dt=case["dt"], cfl=0.5, species=(GAMMA, R_AIR, minf), stream=stream, **opts)
        if kind == "hosted":
            q0 = torch.from_numpy(q).pin_memory()
            out = torch.empty(q0.shape, dtype=torch.float64, pin_memory=True)
        else:
            q0 = torch.tensor(q, dtype=real, device="cuda")
            out = torch.empty_like(q0)
        return {"case": case, "solver": s, "q0": q0, "out": out}
    if kind == "adjoint":
        nodes, bc, ref, q, minf = _adjoint_inputs(case, rng)
        s = Solver(Mesh(nodes), bc, ref, dt="global", cfl=0.5, species=(GAMMA, R_AIR, minf), **opts)
        q0 = torch.tensor(q, dtype=real, device="cuda", requires_grad=True)
        far = torch.tensor(ref[1], dtype=torch.float64, device="cuda", requires_grad=True)
        return {"case": case, "solver": s, "q0": q0, "far": far}
    members = _members(case, rng)
    b = Batch([(Mesh(m[0]), m[1], m[2], m[3]) for m in members], dt="global", cfl=0.5,
              species=(GAMMA, R_AIR, 0.5 if kind == "batch" else 0.3), **opts)
    b.autotune(1)
    if kind == "batch":
        b.capture(case["steps"])
        return {"case": case, "batch": b, "q0": [torch.tensor(m[3], device="cuda") for m in members]}
    return {"case": case, "batch": b,
            "q0": [torch.tensor(m[3], dtype=real, device="cuda", requires_grad=True) for m in members],
            "target": [torch.tensor(m[4], device="cuda") for m in members]}


def run(state):
    from hyperboliconvergence_gb300 import autograd
    case = state["case"]
    kind, n = case["kind"], case["steps"]
    if kind in ("tube", "single"):
        s, out = state["solver"], state["out"]
        s.upload_device(state["q0"])
        s.step(n)
        s.get_state_device(out.data_ptr())
        return out
    if kind == "hosted":
        state["solver"].step_host(state["q0"].numpy(), state["out"].numpy(), n)
        return state["out"]
    if kind == "batch":
        b = state["batch"]
        for k, q in enumerate(state["q0"]):
            b.upload_device(k, q)
        b.replay()
        b.sync()
        # an FP32 batch's states, which the host arrays hold widened
        return torch.cat([torch.from_numpy(b.get_state(k)).to(torch.float32).reshape(-1) for k in range(b.n)])
    if kind == "adjoint":
        q0, far = state["q0"], state["far"]
        cd = autograd.run_objective(state["solver"], q0, [None, far, None, None], n, snapshots=case["snapshots"],
                                    kind="drag", scale=_cd_scale(case["mach"]))
        gq, gf = torch.autograd.grad(cd, [q0, far])
        return {"cd": cd.detach(), "dq0": gq, "dfar": gf}
    q0 = state["q0"]
    loss = autograd.batch_l2_objective(state["batch"], q0, state["target"], n, snapshots=case["snapshots"])
    grads = torch.autograd.grad(loss.sum(), q0)
    return {"loss": loss.detach().to(torch.float32), "dq0": list(grads)}


# ------------------------------------------------------------------------- the work of a pass
STAGES = {"ssp11": 1, "ssp22": 2, "ssp33": 3, "ssp34": 4}
# algorithmic operations of a cell and stage: the two faces' reconstruction and flux and the
# cell's least-squares sums and update (1,114 for Roe + van Albada by the oracle's tally)
FLOPS = {"roe": 1114.0, "slau": 900.0, "ausmpup": 1000.0, "rusanov": 700.0}


def work(case):
    kind = case["kind"]
    real = 4 if case["precision"] == "fp32" else 8
    st = STAGES[case["rk"]] * case["steps"]
    if kind == "tube":
        cells, nv, flops = case["nc"], 3, 0.45 * FLOPS[case["flux"]]
    elif kind in ("batch", "badjoint"):
        sizes = np.random.default_rng(case["lo"] * 7919 + case["hi"] * 31 + case["n"])
        of, cells, nv, flops = case["of"], 0, 4, FLOPS[case["flux"]]
        for _ in range(case["n"]):
            a, b = (int(v) * of for v in sizes.integers(-(-case["lo"] // of), case["hi"] // of + 1, 2))
            cells += a * b if kind == "batch" else a * a
    else:
        cells, nv, flops = case["ni"] * case["nj"], 4, FLOPS[case["flux"]]
    # a stage reads the stage state and the step's start, writes the next, and reads the volume
    # and one metric value; the reverse of a stage costs twice the stage
    per, times = (3 * nv + 2) * real, 3.0 if kind in ("adjoint", "badjoint") else 1.0
    return {"bytes": times * cells * st * per, "flops": times * cells * st * flops}


# ------------------------------------------------------------------------- exact: plain torch float64
TABLES = {
    "ssp22": ([[1.0], [0.5, 0.5]], [1.0, 1.0]),
    "ssp33": ([[1.0], [0.5, 0.5], [1 / 6, 1 / 6, 2 / 3]], [1.0, 0.5, 1.0]),
    "ssp34": ([[1.0], [0.5, 0.5], [1 / 3, 1 / 3, 1 / 3], [1 / 6, 1 / 6, 1 / 6, 0.5]], [0.5, 1.0, 0.5, 1.0]),
}


def _limit(kind, a, b):
    zero = torch.zeros((), dtype=a.dtype, device=a.device)
    if kind == "nolimit3":
        return (2.0 * a + b) / 3.0
    if kind == "vanalbada":
        den = a * a + b * b
        on = (a * b > 0) & (den > 0)
        return torch.where(on, a * b * (a + b) / torch.where(on, den, zero + 1.0), zero)
    if kind == "vanleer":
        den = a.abs() + b.abs()
        return torch.where(den > 0, (a * b.abs() + a.abs() * b) / torch.where(den > 0, den, zero + 1.0), zero)
    if kind == "minmod":
        return torch.where(a > 0, torch.minimum(a, torch.maximum(b, zero)), torch.maximum(a, torch.minimum(b, zero)))
    up = torch.maximum(zero, torch.minimum(0.5 * (a + b), torch.minimum(2 * b, 2 * a)))  # mc
    return torch.where(a > 0, up, torch.minimum(zero, torch.maximum(0.5 * (a + b), torch.maximum(2 * b, 2 * a))))


class _State:
    def __init__(self, q):
        self.u, self.v, self.r, self.p = q
        k = 0.5 * (self.u ** 2 + self.v ** 2)
        self.a2 = GAMMA * self.p / self.r
        self.a = self.a2.sqrt()
        self.h = self.a2 / (GAMMA - 1.0) + k

    def cons(self):
        return [self.r * self.u, self.r * self.v, self.r, self.r * self.h - self.p]


def _roe_average(l, r):
    cr = (r.r / l.r).sqrt()
    wl = 1.0 / (1.0 + cr)
    wr = 1.0 - wl
    u, v, h = wl * l.u + wr * r.u, wl * l.v + wr * r.v, wl * l.h + wr * r.h
    k = 0.5 * (u * u + v * v)
    return cr, u, v, h, k, (GAMMA - 1.0) * (h - k)


def _flux(kind, minf, nx, ny, area, ql, qr):
    """Interface flux times the area (4 components) and the spectral radius times the area."""
    l, r = _State(ql), _State(qr)
    ul, ur = nx * l.u + ny * l.v, nx * r.u + ny * r.v
    if kind in ("roe", "rusanov"):
        f = [0.0] * 4
        for s, un in ((l, ul), (r, ur)):
            m = s.r * un
            f = [a + b for a, b in zip(f, (m * s.u + s.p * nx, m * s.v + s.p * ny, m, m * s.h))]
        lam = torch.maximum(ul.abs() + l.a, ur.abs() + r.a)
        d = [b - a for a, b in zip(l.cons(), r.cons())]
        if kind == "rusanov":
            return torch.stack([0.5 * area * (a - lam * b) for a, b in zip(f, d)]), lam * area
        # the reference's Roe: the jump in the face frame, the averaged velocity in the global one
        cr, ua, va, _, ka, a2 = _roe_average(l, r)
        ra, aa = cr * l.r, a2.sqrt()
        un = nx * ua + ny * va
        wave = [un.abs()]
        for s in (-1.0, 1.0):
            x, xl, xr = un + s * aa, ul + s * l.a, ur + s * r.a
            e = 0.05 * torch.clamp(torch.maximum(x - xl, xr - x), min=0.0)
            ax = x.abs()
            fix = ax <= e
            wave.append(torch.where(fix, 0.5 * (e + ax * ax / torch.where(fix & (e > 0), e, torch.ones_like(e))), ax))
        c0, c1 = nx * d[0] + ny * d[1], nx * d[1] - ny * d[0]
        du0, du1 = (c0 - ua * d[2]) / ra, (c1 - va * d[2]) / ra
        dp = (GAMMA - 1.0) * (ka * d[2] + d[3] - ua * c0 - va * c1)
        w0 = wave[0] * GAMMA * (dp / a2 - d[2]) / ra
        w1 = wave[1] * (du0 - dp / (ra * aa))
        w2 = wave[2] * (du0 + dp / (ra * aa))
        w3 = wave[0] * du1
        dpp = 0.5 * ra * aa * (w2 - w1)
        dr = dpp / a2 - ra * w0 / GAMMA
        du = 0.5 * (w1 + w2)
        e0, e1 = ra * du + ua * dr, ra * w3 + va * dr
        e3 = dpp / (GAMMA - 1.0) + ra * (ua * du + va * w3) + ka * dr
        diss = [nx * e0 - ny * e1, ny * e0 + nx * e1, dr, e3]
        return (torch.stack([0.5 * area * (a - b) for a, b in zip(f, diss)]),
                torch.maximum(lam, un.abs() + aa) * area)

    def m2(s, m):
        return s * 0.25 * (m + s) ** 2

    dp = r.p - l.p
    one = torch.ones_like(dp)
    if kind == "slau":
        ua = (0.5 * (l.u ** 2 + l.v ** 2 + r.u ** 2 + r.v ** 2)).sqrt()
        aa = 0.5 * (l.a + r.a)
        ma = ua / aa
        ml, mr = ul / aa, ur / aa
        una = (l.r * ul.abs() + r.r * ur.abs()) / (l.r + r.r)
        chi = (1.0 - torch.clamp(ma, max=1.0)) ** 2
        g = -torch.clamp(torch.clamp(ml, max=0.0), min=-1.0) * torch.clamp(torch.clamp(mr, min=0.0), max=1.0)
        mdot = 0.5 * ((l.r * ul + r.r * ur - una * (r.r - l.r)) * (1.0 - g) - chi * dp / aa) * area
        bl = torch.where(ml.abs() > 1.0, one, m2(1.0, ml) * (2.0 - ml))
        br = torch.where(mr.abs() > 1.0, one, m2(-1.0, mr) * (-2.0 - mr))
        pa = 0.5 * ((l.p + r.p) - (bl - br) * dp + ma * (bl + br - 1.0) * (l.p + r.p)) * area
        lam = torch.maximum(l.a, r.a) + torch.maximum(ul.abs(), ur.abs())
    else:  # AUSM+up, convective scalings
        c = 2.0 * (GAMMA - 1.0) / (GAMMA + 1.0)
        sl, sr = c * l.h, c * r.h
        als, ars = sl / torch.maximum(ul, sl.sqrt()), sr / torch.maximum(-ur, sr.sqrt())
        ra, a = 0.5 * (l.r + r.r), torch.minimum(als, ars)
        ml, mr = ul / a, ur / a
        m0 = (0.5 * (ml * ml + mr * mr)).sqrt()
        m0c = torch.clamp(torch.clamp(m0, min=minf), max=1.0)
        fa = m0c * (2.0 - m0c)
        lsup, rsup = ml.abs() > 1.0, mr.abs() > 1.0
        mlp = torch.where(lsup, 0.5 * (ml + ml.abs()), m2(1.0, ml) * (1.0 - 2.0 * m2(-1.0, ml)))
        mrm = torch.where(rsup, 0.5 * (mr - mr.abs()), m2(-1.0, mr) * (1.0 + 2.0 * m2(1.0, mr)))
        mp = 0.25 * torch.clamp(1.0 - m0 * m0, min=0.0) * dp / (fa * ra * a * a)
        uf = a * (mlp + mrm - mp) * area
        alpha = 0.1875 * (5.0 * fa * fa - 4.0)
        plp = torch.where(lsup, one, m2(1.0, ml) * (2.0 - ml) - 16.0 * alpha * ml * m2(1.0, ml) * m2(-1.0, ml))
        prm = torch.where(rsup, one, m2(-1.0, mr) * (-2.0 - mr) + 16.0 * alpha * mr * m2(-1.0, mr) * m2(1.0, mr))
        pu = 1.5 * plp * prm * ra * (fa * a) * (ur - ul)
        pa = (plp * l.p + prm * r.p - pu) * area
        mdot = uf * torch.where(uf > 0, l.r, r.r)
        amax = torch.maximum(a * a, torch.maximum(l.a2, r.a2)).sqrt()
        lam = 0.5 * (m0c + 1.0) / fa * amax + torch.maximum(uf.abs(), torch.maximum(ul.abs(), ur.abs()))
    left = mdot > 0
    return (torch.stack([mdot * torch.where(left, l.u, r.u) + pa * nx, mdot * torch.where(left, l.v, r.v) + pa * ny,
                         mdot, mdot * torch.where(left, l.h, r.h)]), lam * area)


def _riemann(nx, ny, qi, qf):
    """Riemann-invariant far field, (nx, ny) into the domain: the ghost state."""
    def rot(q):
        return torch.stack([nx * q[0] + ny * q[1], nx * q[1] - ny * q[0], q[2], q[3]])
    i, f = _State(rot(qi)), _State(rot(qf))
    _, ua, va, _, _, a2 = _roe_average(i, f)
    inflow = ua > 0
    rim, rip = i.u - 2.0 * i.a / (GAMMA - 1.0), f.u + 2.0 * f.a / (GAMMA - 1.0)
    ub, ab = 0.5 * (rim + rip), 0.25 * (GAMMA - 1.0) * (rip - rim)
    s = torch.where(inflow, f.a2, i.a2) / (GAMMA * torch.where(inflow, f.r, i.r) ** (GAMMA - 1.0))
    rb = (ab * ab / (GAMMA * s)) ** (1.0 / (GAMMA - 1.0))
    vt = torch.where(inflow, f.v, i.v)
    sub = torch.stack([nx * ub - ny * vt, ny * ub + nx * vt, rb, rb * ab * ab / GAMMA])
    out = torch.where((ua / a2.sqrt()).abs() > 1.0, torch.where(inflow, qf, qi), sub)
    return torch.where(ua / (ua * ua + va * va).sqrt() < 0.001, qi, out)


class _Direction:
    """Face geometry of one grid direction (faces along the first axis of the given arrays)."""

    def __init__(self, x, c, periodic, flip):
        # x: nodes (2, n+1, m+1), c: cell centres (2, n, m), first axis across the faces
        p0, p1 = (x[:, :, 1:], x[:, :, :-1]) if flip else (x[:, :, :-1], x[:, :, 1:])
        if periodic:
            p0, p1 = (torch.cat([p[:, :-1], p[:, :1]], 1) for p in (p0, p1))
        t = p0 - p1
        self.area = t.square().sum(0).sqrt()
        self.nx, self.ny = -t[1] / self.area, t[0] / self.area
        self.centre = fc = 0.5 * (p0 + p1)
        self.periodic = periodic
        if periodic:
            shift = 0.5 * ((x[:, -1, :-1] - x[:, 0, :-1]) + (x[:, -1, 1:] - x[:, 0, 1:]))
            cl = torch.cat([(c[:, -1] - shift)[:, None], c[:, :-1]], 1)
            self.d = c - cl  # faces 0..n-1
            f = fc[:, :-1]
            self.dl, self.dr = (f - cl).square().sum(0).sqrt(), (c - f).square().sum(0).sqrt()
        else:
            self.d = c[:, 1:] - c[:, :-1]  # faces 1..n-1
            f = fc[:, 1:-1]
            self.dl, self.dr = (f - c[:, :-1]).square().sum(0).sqrt(), (c[:, 1:] - f).square().sum(0).sqrt()
            self.mirror = [c[:, 0] - c[:, 1], c[:, -1] - c[:, -2]]

    def scatter(self, t):
        """Sum of a face quantity (..., faces, m) over the two cells of each pair face."""
        if self.periodic:
            return t + torch.roll(t, -1, -2)
        zero = torch.zeros_like(t[..., :1, :])
        return torch.cat([zero, t], -2) + torch.cat([t, zero], -2)


def _solve(x, d):
    """x^-1 d of symmetric 2x2 metrics x = (xx, xy, yy)."""
    det = 1.0 / (x[0] * x[2] - x[1] * x[1])
    return torch.stack([det * (x[2] * d[0] - x[1] * d[1]), det * (x[0] * d[1] - x[1] * d[0])])


class _Mesh2D:
    def __init__(self, nodes, bc, ref, minf, case):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        p = torch.tensor(nodes, dtype=torch.float64, device=dev).permute(2, 0, 1)
        self.case, self.minf, self.bc = case, minf, bc
        self.ref = [None if r is None else r if torch.is_tensor(r) else
                    torch.tensor(np.ascontiguousarray(r), dtype=torch.float64, device=dev) for r in ref or [None] * 4]
        a, b, c, d = p[:, :-1, :-1], p[:, 1:, :-1], p[:, :-1, 1:], p[:, 1:, 1:]
        ti, tj = 0.25 * (b + d - a - c), 0.25 * (c + d - a - b)
        self.vol = (ti[0] * tj[1] - ti[1] * tj[0]).abs()
        ctr = 0.25 * (a + b + c + d)
        self.dirs = [_Direction(p, ctr, bc[0] == "periodic", False),
                     _Direction(p.transpose(1, 2), ctr.transpose(1, 2), bc[2] == "periodic", True)]
        self.xm = 0.0
        for k, g in enumerate(self.dirs):
            x = g.scatter(torch.stack([g.d[0] ** 2, g.d[0] * g.d[1], g.d[1] ** 2]))
            if not g.periodic:
                x = x.clone()
                for end, m in zip((0, -1), g.mirror):
                    x[:, end] += torch.stack([m[0] ** 2, m[0] * m[1], m[1] ** 2])
            self.xm = self.xm + (x if k == 0 else x.transpose(1, 2))
        for k, g in enumerate(self.dirs):
            xm = self.xm if k == 0 else self.xm.transpose(1, 2)
            dd = torch.stack([g.d[0] ** 2, g.d[0] * g.d[1], g.d[1] ** 2])
            n = torch.stack([g.nx, g.ny])
            xl, xr, n = (torch.roll(xm, 1, 1), xm, n[:, :-1]) if g.periodic else (xm[:, :-1], xm[:, 1:], n[:, 1:-1])
            g.wl, g.wr = _solve(xl - dd, n), _solve(xr - dd, n)
            if not g.periodic:
                g.end = []
                for end, m, c in zip((0, -1), g.mirror, (ctr if k == 0 else ctr.transpose(1, 2))[:, (0, -1)].unbind(1)):
                    mm = torch.stack([m[0] ** 2, m[0] * m[1], m[1] ** 2])
                    f = g.centre[:, end]
                    nn = torch.stack([g.nx[end], g.ny[end]])
                    g.end.append(((c - f).square().sum(0).sqrt(), _solve(xm[:, end] - mm, nn),
                                  _solve(xm[:, end], c - f)))

    def gradients(self, q):
        m = 0.0
        for k, g in enumerate(self.dirs):
            y = q if k == 0 else q.transpose(1, 2)
            dq = y - torch.roll(y, 1, 1) if g.periodic else y[:, 1:] - y[:, :-1]
            t = g.scatter(dq[:, None] * g.d[None])
            m = m + (t if k == 0 else t.transpose(2, 3))
        return m

    def residual(self, q):
        lim, flux = self.case["limiter"], self.case["flux"]
        qm = self.gradients(q)
        res, lam = 0.0, 0.0
        for k, g in enumerate(self.dirs):
            y, m = (q, qm) if k == 0 else (q.transpose(1, 2), qm.transpose(2, 3))
            if g.periodic:
                yl, yr, ml, mr = torch.roll(y, 1, 1), y, torch.roll(m, 1, 2), m
                nx, ny, area = g.nx[:-1], g.ny[:-1], g.area[:-1]
            else:
                yl, yr, ml, mr = y[:, :-1], y[:, 1:], m[:, :, :-1], m[:, :, 1:]
                nx, ny, area = g.nx[1:-1], g.ny[1:-1], g.area[1:-1]
            dq = yr - yl
            gc = dq / (g.dl + g.dr)
            gl = (ml * g.wl).sum(1) - dq * (g.d * g.wl).sum(0)
            gr = (mr * g.wr).sum(1) - dq * (g.d * g.wr).sum(0)
            f, fl = _flux(flux, self.minf, nx, ny, area, yl + g.dl * _limit(lim, gc, gl),
                          yr - g.dr * _limit(lim, gc, gr))
            if g.periodic:
                f, fl = torch.cat([f, f[:, :1]], 1), torch.cat([fl, fl[:1]], 0)
            else:
                ends = [self.boundary(2 * k + e, g, e, y, m) for e in (0, 1)]
                f = torch.cat([ends[0][0][:, None], f, ends[1][0][:, None]], 1)
                fl = torch.cat([ends[0][1][None], fl, ends[1][1][None]], 0)
            r, s = f[:, :-1] - f[:, 1:], fl[:-1] + fl[1:]
            res, lam = res + (r if k == 0 else r.transpose(1, 2)), lam + (s if k == 0 else s.t())
        return res, lam

    def wall_pressure(self, side, y, m):
        d = self.dirs[side // 2]
        e = side % 2
        at = -1 if e else 0
        return y[:, at] - (m[:, :, at] * d.end[e][2]).sum(1)

    def boundary(self, side, g, e, y, m):
        at = -1 if e else 0
        qi, mi = y[:, at], m[:, :, at]
        nx, ny, area = g.nx[at], g.ny[at], g.area[at]
        if self.bc[side] == "wall":
            w = _State(self.wall_pressure(side, y, m))
            zero = torch.zeros_like(w.p)
            un = nx * w.u + ny * w.v
            return torch.stack([area * w.p * nx, area * w.p * ny, zero, zero]), area * (un.abs() + w.a)
        sign = -1.0 if e else 1.0
        qg = self.ref[side] if self.bc[side] == "fixed" else _riemann(sign * nx, sign * ny, qi, self.ref[side])
        dist, w, _ = g.end[e]
        dq = sign * (qi - qg)
        s = dist * _limit(self.case["limiter"], dq / (2.0 * dist), (mi * w).sum(1))
        ql, qr = (qi + s, qg) if e else (qg, qi - s)
        return _flux(self.case["flux"], self.minf, nx, ny, area, ql, qr)

    def drag(self, q):
        """Pressure force along x on the wall at side 0."""
        g = self.dirs[0]
        p = self.wall_pressure(0, q, self.gradients(q))[3]
        return -(g.area[0] * p * g.nx[0]).sum()

    def steps(self, q, n, cfl, mode, each=None):
        alpha, beta = TABLES[self.case["rk"]]
        for _ in range(n):
            kept, q0, qs = [], q, q
            for a, b in zip(alpha, beta):
                r, lam = self.residual(qs)
                if not kept:
                    with torch.no_grad():
                        if mode == "local":
                            dt_v = cfl / lam
                        else:
                            dt_v = cfl / (lam / self.vol).max() / self.vol
                kept.append(r)
                tot = sum(c * x for c, x in zip(a, kept)) * (b * dt_v)
                c = [x + y for x, y in zip(_State(q0).cons(), tot)]
                u, v = c[0] / c[2], c[1] / c[2]
                qs = torch.stack([u, v, c[2], (GAMMA - 1.0) * (c[3] - 0.5 * c[2] * (u * u + v * v))])
            q = qs
            if each is not None:
                each(q)
        return q


def _tube_exact(case, x, ref, q):
    """The 1D path: cells between nodes x, Riemann far fields at both ends."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    x, ref, q = t(x), [t(r) for r in ref], t(q)
    c, vol = 0.5 * (x[:-1] + x[1:]), x[1:] - x[:-1]
    d = c[1:] - c[:-1]
    xm = torch.zeros_like(c)
    xm[1:] += d * d
    xm[:-1] += d * d
    xm[0] += d[0] ** 2
    xm[-1] += d[-1] ** 2
    dl, dr = x[1:-1] - c[:-1], c[1:] - x[1:-1]
    wl, wr = 1.0 / (xm[:-1] - d * d), 1.0 / (xm[1:] - d * d)
    lim, one = case["limiter"], torch.ones((), dtype=torch.float64, device=dev)

    def four(v):
        return torch.stack([v[0], torch.zeros_like(v[0]), v[1], v[2]])

    def flux(a, b):
        f, lam = _flux(case["flux"], 1e-4, one, 0.0 * one, one, four(a), four(b))
        return f[[0, 2, 3]], lam

    def residual(y):
        dq = y[:, 1:] - y[:, :-1]
        m = torch.zeros_like(y)
        m[:, 1:] += dq * d
        m[:, :-1] += dq * d
        gc = dq / (dl + dr)
        f, lam = flux(y[:, :-1] + dl * _limit(lim, gc, m[:, :-1] * wl - dq * d * wl),
                      y[:, 1:] - dr * _limit(lim, gc, m[:, 1:] * wr - dq * d * wr))
        ends = []
        for e in (0, 1):
            at, sign = (-1, -1.0) if e else (0, 1.0)
            qi = y[:, at:][:, :1] if e else y[:, :1]
            g4 = _riemann(sign * one, 0.0 * one, four(qi), four(ref[e][:, None]))
            qg = g4[[0, 2, 3]]
            dist = (x[at] - c[at]).abs()
            w = 1.0 / (xm[at] - (c[0] - c[1] if not e else c[-1] - c[-2]) ** 2)
            s = dist * _limit(lim, sign * (qi - qg) / (2.0 * dist), (m[:, -1:] if e else m[:, :1]) * w)
            ends.append(flux(qi + s, qg) if e else flux(qg, qi - s))
        f = torch.cat([ends[0][0], f, ends[1][0]], 1)
        lam = torch.cat([ends[0][1], lam, ends[1][1]])
        return f[:, :-1] - f[:, 1:], lam[:-1] + lam[1:]

    alpha, beta = TABLES[case["rk"]]
    for _ in range(case["steps"]):
        kept, y = [], q
        for a, b in zip(alpha, beta):
            r, lam = residual(y)
            if not kept:
                dt_v = 0.8 / (lam / vol).max() / vol
            kept.append(r)
            u, rho, p = q
            tot = sum(k * v for k, v in zip(a, kept)) * (b * dt_v)
            m, rho1, en = rho * u + tot[0], rho + tot[1], p / (GAMMA - 1.0) + 0.5 * rho * u * u + tot[2]
            y = torch.stack([m / rho1, rho1, (GAMMA - 1.0) * (en - 0.5 * m * m / rho1)])
        q = y
    return q


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    narrow = (lambda q: q.astype(np.float32).astype(np.float64)) if case["precision"] == "fp32" else (lambda q: q)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "tube":
        x, ref, q = _tube_inputs(case, rng)
        return _tube_exact(case, x, ref, narrow(q))
    if kind in ("single", "hosted"):
        nodes, bc, ref, q, minf = _mesh_inputs(case, rng)
        with torch.no_grad():
            return _Mesh2D(nodes, bc, ref, minf, case).steps(torch.tensor(narrow(q), device=dev), case["steps"], 0.5,
                                                             case["dt"])
    if kind == "adjoint":
        nodes, bc, ref, q, minf = _adjoint_inputs(case, rng)
        q0 = torch.tensor(q, device=dev, requires_grad=True)
        far = torch.tensor(ref[1], device=dev, requires_grad=True)
        m = _Mesh2D(nodes, bc, [None, far, None, None], minf, case)
        force = []
        m.steps(q0, case["steps"], 0.5, "global", lambda y: force.append(m.drag(y)))
        cd = _cd_scale(case["mach"]) * sum(force) / case["steps"]
        gq, gf = torch.autograd.grad(cd, [q0, far])
        return {"cd": cd.detach(), "dq0": gq, "dfar": gf}
    members = _members(case, rng)
    if kind == "batch":
        out = []
        with torch.no_grad():
            for nodes, bc, ref, q, _ in members:
                m = _Mesh2D(nodes, bc, ref, 0.5, case)
                out.append(m.steps(torch.tensor(narrow(q), device=dev), case["steps"], 0.5, "global").reshape(-1))
        return torch.cat(out)
    loss, grads = [], []
    for nodes, bc, _, q, target in members:
        m = _Mesh2D(nodes, bc, None, 0.3, case)
        q0 = torch.tensor(narrow(q), device=dev, requires_grad=True)
        j = (m.steps(q0, case["steps"], 0.5, "global") - torch.tensor(target, device=dev)).square().sum()
        grads.append(torch.autograd.grad(j, q0)[0])
        loss.append(j.detach())
    return {"loss": torch.stack(loss), "dq0": grads}
