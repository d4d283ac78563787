"""Workloads by which the framework's speed is measured, through its public entry points.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more of
the same ranges, ``prepare(case, seed)`` what a program has in hand before the call, ``run(state)``
one pass, ``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the outputs of a pass in 64 bits from a plain torch statement of the method
(None where there is none or it would take too long).

Kinds of case:
  step      Simulation: load moments, advance some steps, read the state back
  dropin    GpuSimulator in a fixed periodic box: some steps, then its two state arrays
  pulse     GpuSimulator on host arrays: construction, steps, moments()
  gradient  rollout forward and backward (inverse problem)
  lbm       HexLBM steps
  fields    bin_fields_device / bin_fields3_device
  stages    disperse, create_control_points, refine_control_points, resample
"""

import itertools
import math
import random

import numpy as np
import torch

from direbm_gb300 import fields as dbm_fields
from direbm_gb300.adjoint import Tape, rollout
from direbm_gb300.lbm import HexLBM
from direbm_gb300.sim import Instance, Simulation
from direbm_gb300.warp import (GpuSimulator, create_control_points, disperse, refine_control_points,
                               resample)

DEV = "cuda"


def listed():
    return [
        # the headline: a batch of independent 2D runs of 4k-256k points, state resident, float32
        # moments in and out without a host wait
        _step("ensemble", "D2Q9", "fp32dev", members=256, lo=64, hi=512, steps=4, presorted=True, pipelined=True),
        # one small box: the shortest steps, where latency and launches count
        _step("box2d_small", "D2Q9", "fp32dev", nx=64, ny=64, steps=10),
        # the Taylor-Green box of the double-precision checks
        _step("box2d_fp64", "D2Q9", "fp64", nx=128, ny=128, steps=2),
        # flow past a bounce-back sphere with an inflow layer, about 2 M points
        _step("sphere", "D3Q19", "fp32dev", nx=160, ny=112, nz=112, steps=2, obstacle=True),
        # a 3D box in double precision
        _step("box3d_fp64", "D3Q19", "fp64", nx=44, ny=40, nz=37, steps=1),
        # the drop-in simulator at the reference's parameters (D2Q7, r = dx, cell dx / 4), saturated
        {"name": "dropin_flow", "kind": "dropin", "precision": "fp32dev", "nx": 160, "ny": 144, "steps": 4},
        # the reference's own example: a block at rest with a density pulse, from and to host arrays
        {"name": "dropin_pulse", "kind": "pulse", "precision": "fp32dev", "half": 6, "steps": 16},
        # the inverse problem: 64k points, checkpointed rollout and its gradient
        {"name": "gradient", "kind": "gradient", "precision": "fp32dev", "n": 256, "steps": 10, "every": 5},
        # hexagonal lattice Boltzmann: eight runs of the 1024 x 1024 shear wave, and one smaller in
        # double precision
        {"name": "hex_lbm", "kind": "lbm", "precision": "fp32dev", "ni": 1024, "nj": 1024, "runs": 8, "steps": 10},
        {"name": "hex_lbm_fp64", "kind": "lbm", "precision": "fp64", "ni": 1024, "nj": 768, "runs": 2, "steps": 4},
        # macroscopic fields of a state for plots and statistics: 4 x 4-cell bins
        {"name": "fields", "kind": "fields", "lattice": "D2Q9", "n": 1280, "bin": 4.0},
        # the four propagation stages on explicit arrays
        {"name": "stages", "kind": "stages", "n": 192},
    ]


def _step(name, lattice, precision, members=1, lo=0, hi=0, nx=0, ny=0, nz=0, steps=1, obstacle=False, soft=False,
          presorted=False, pipelined=False):
    c = {"name": name, "kind": "step", "lattice": lattice, "precision": precision, "members": members, "lo": lo,
         "hi": hi, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "obstacle": obstacle, "soft": soft,
         "presorted": presorted, "pipelined": pipelined}
    return c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ensemble", "box2d", "box2d", "box2d_fp64", "sphere", "box3d", "dropin", "pulse", "gradient",
                       "lbm", "fields", "stages"])
    if kind == "ensemble":
        c = _step("", "D2Q9", "fp32dev", members=_log(rng, 5, 250), lo=48, hi=_log(rng, 100, 500),
                  steps=rng.randint(1, 4), presorted=rng.random() < 0.5, pipelined=rng.random() < 0.5)
    elif kind == "box2d":
        lat = rng.choice(["D2Q9", "D2Q9", "D2Q7"])
        c = _step("", lat, "fp32dev", nx=_log(rng, 24, 1500), ny=_log(rng, 24, 1500), steps=rng.randint(1, 10),
                  soft=lat == "D2Q7" and rng.random() < 0.3, presorted=rng.random() < 0.5)
    elif kind == "box2d_fp64":
        c = _step("", rng.choice(["D2Q9", "D2Q7"]), "fp64", nx=_log(rng, 24, 300), ny=_log(rng, 24, 300),
                  steps=rng.randint(1, 3))
    elif kind == "sphere":
        c = _step("", "D3Q19", "fp32dev", nx=rng.randint(64, 160), ny=rng.randint(56, 112), nz=rng.randint(56, 112),
                  steps=rng.randint(1, 2), obstacle=True)
    elif kind == "box3d":
        fp64 = rng.random() < 0.4
        top = 48 if fp64 else 110
        c = _step("", rng.choice(["D3Q19", "D3Q19", "D3Q13"]), "fp64" if fp64 else "fp32dev", nx=_log(rng, 16, top),
                  ny=_log(rng, 16, top), nz=_log(rng, 16, top), steps=1)
    elif kind == "dropin":
        c = {"kind": "dropin", "precision": rng.choice(["fp32dev", "fp32dev", "fp64"]), "nx": _log(rng, 12, 160),
             "ny": _log(rng, 12, 160), "steps": rng.randint(1, 4)}
        if c["precision"] == "fp64":
            c["nx"], c["ny"], c["steps"] = min(c["nx"], 40), min(c["ny"], 40), 1
    elif kind == "pulse":
        c = {"kind": "pulse", "precision": "fp32dev", "half": _log(rng, 3, 40), "steps": rng.randint(4, 20)}
    elif kind == "gradient":
        c = {"kind": "gradient", "precision": rng.choice(["fp32dev", "fp32dev", "fp64"]), "n": _log(rng, 24, 300),
             "steps": rng.randint(2, 10), "every": rng.randint(2, 5)}
        if c["precision"] == "fp64":
            c["n"], c["steps"] = min(c["n"], 96), min(c["steps"], 3)
    elif kind == "lbm":
        c = {"kind": "lbm", "precision": rng.choice(["fp32dev", "fp64"]), "ni": _log(rng, 33, 1100),
             "nj": _log(rng, 33, 1100), "runs": rng.randint(1, 8), "steps": rng.randint(1, 10)}
        if c["precision"] == "fp64":
            c["runs"] = min(c["runs"], 3)
    elif kind == "fields":
        c = {"kind": "fields", "lattice": rng.choice(["D2Q9", "D2Q7", "D3Q19"]), "n": _log(rng, 90, 1500),
             "bin": round(rng.uniform(1.0, 8.0), 2)}
        if c["lattice"] == "D3Q19":
            c["n"] = max(12, int(c["n"] ** 0.66))
    else:
        c = {"kind": "stages", "n": _log(rng, 24, 260)}
    c.pop("name", None)
    return c


# ---- velocity sets and inputs -----------------------------------------------------------------------


def _lattice(name):
    s = math.sqrt(3.0) / 2.0
    if name == "D2Q7":
        C = [[0, 0], [1, 0], [0.5, s], [-0.5, s], [-1, 0], [-0.5, -s], [0.5, -s]]
        W, cs2 = [0.5] + [1 / 12] * 6, 0.25
    elif name == "D2Q9":
        C = [[0, 0], [1, 0], [0, 1], [-1, 0], [0, -1], [1, 1], [-1, 1], [-1, -1], [1, -1]]
        W, cs2 = [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4, 1 / 3
    elif name == "D3Q13":
        p = (1 + math.sqrt(5.0)) / 2
        ico = [[0, 1, p], [0, 1, -p], [0, -1, p], [0, -1, -p], [1, p, 0], [1, -p, 0], [-1, p, 0], [-1, -p, 0],
               [p, 0, 1], [p, 0, -1], [-p, 0, 1], [-p, 0, -1]]
        n = math.sqrt(1 + p * p)
        C = [[0, 0, 0]] + [[v / n for v in r] for r in ico]
        W, cs2 = [2 / 5] + [1 / 20] * 12, 0.2
    else:
        C = [[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0],
             [1, -1, 0], [-1, 1, 0], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1], [0, 1, 1], [0, -1, -1],
             [0, 1, -1], [0, -1, 1]]
        W, cs2 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, 1 / 3
    t = {"dtype": torch.float64, "device": DEV}
    return torch.tensor(C, **t), torch.tensor(W, **t), cs2


def _feq(rho, u, C, W, cs2):
    cu = u @ C.T
    br = 1 + cu / cs2 + cu * cu / (2 * cs2 * cs2) - (u * u).sum(-1, keepdim=True) / (2 * cs2)
    return rho[..., None] * W * br


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _grid(dims, g, spacing=1.0):
    """One jittered point per cell of a box, row by row (x fastest)."""
    axes = [torch.arange(n, dtype=torch.float64, device=DEV) for n in dims]
    mesh = torch.meshgrid(*axes[::-1], indexing="ij")[::-1]
    x = torch.stack([m.reshape(-1) for m in mesh], 1) + 0.5
    return (x + (torch.rand(x.shape, generator=g, dtype=torch.float64, device=DEV) - 0.5) * 0.5) * spacing


def _modes(x, size, g, rms=0.02, modes=8):
    """Velocity of random Fourier modes with wave numbers up to 4, divergence-free in 2D."""
    D = x.shape[1]
    r = torch.rand((modes, 3 * D + 2), generator=g, dtype=torch.float64, device=DEV).cpu()
    u = torch.zeros_like(x)
    for row in r:
        k = torch.floor(row[:D] * 9) - 4
        if not bool(k.any()):
            k[0] = 1.0
        e = torch.tensor([-k[1], k[0]]) if D == 2 else torch.linalg.cross(k, row[D:2 * D] - 0.5 + 1e-3)
        e = (e / torch.linalg.norm(e)).to(x)
        phase = (x / torch.tensor(size, dtype=x.dtype, device=DEV)) @ k.to(x) * (2 * math.pi)
        u += (row[-1].item() - 0.5) * e * torch.sin(phase + 2 * math.pi * row[-2].item())[:, None]
    return u * (rms / torch.sqrt((u * u).sum(1).mean()))


def _boxes(case):
    """(dims, tau) of every box of a step case; sizes belong to the case, not to the seed."""
    D = 3 if case["lattice"].startswith("D3") else 2
    r = random.Random(1)
    if case["members"] == 1:
        return [((case["nx"], case["ny"], case["nz"])[:D], 0.56 if case["obstacle"] else 0.6)]
    return [((_log(r, case["lo"], case["hi"]),) * 2, r.uniform(0.55, 1.0)) for _ in range(case["members"])]


def _sphere(dims):
    radius = min(dims) / 7.0
    return (dims[0] * 0.35, dims[1] * 0.5, dims[2] * 0.5), radius


def _step_inputs(case, seed):
    """(instance, position, f) of a step case in float64, the sizes of its boxes, dx, r, cell."""
    g = _generator(seed)
    C, W, cs2 = _lattice(case["lattice"])
    inst, pos, f = [], [], []
    for i, (dims, _) in enumerate(_boxes(case)):
        x = _grid(dims, g)
        if case["obstacle"]:
            c, r = _sphere(dims)
            x = x[((x - torch.tensor(c, dtype=x.dtype, device=DEV)) ** 2).sum(1) >= (r + 0.5) ** 2]
            u = torch.zeros_like(x)
            u[:, 0] = 0.04
            u += _modes(x, dims, g, rms=0.004)
        else:
            u = _modes(x, dims, g)
        inst.append(torch.full((len(x),), i, dtype=torch.int32, device=DEV))
        pos.append(x)
        f.append(_feq(torch.ones(len(x), dtype=x.dtype, device=DEV), u, C, W, cs2))
    return torch.cat(inst), torch.cat(pos), torch.cat(f)


def _in_precision(case, *arrays):
    dt = torch.float32 if case["precision"] == "fp32dev" else torch.float64
    return tuple(a.to(dt) for a in arrays)


def _rows(a, n):
    """An array whose row count depends on the moments, in the fixed frame of n rows it is stored in."""
    if len(a) >= n:
        return a
    if isinstance(a, torch.Tensor):
        return torch.nn.functional.pad(a, (0, 0, 0, n - len(a)))
    return np.pad(a, ((0, n - len(a)), (0, 0)))


def _r_res(case):
    return 1.02 if case["soft"] else 1.5


# ---- prepare and run ----------------------------------------------------------------------------------


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _prepare_step(case, seed):
    inst, pos, f = _step_inputs(case, seed)
    pos, f = _in_precision(case, pos, f)
    boxes = []
    for dims, tau in _boxes(case):
        extra = {"obstacle": _sphere(dims), "inflow": ((0.04, 0.0, 0.0), 2)} if case["obstacle"] else {}
        boxes.append(Instance(dims=dims, tau=tau, **extra))
    cap = int(1.2 * math.prod(boxes[0].dims)) if case["obstacle"] else 0
    sim = Simulation(boxes, lattice=case["lattice"], precision=case["precision"], dx=1.0, r_res=_r_res(case), cell=1.0,
                     moment_capacity=cap, kappa_soft=5 if case["soft"] else 0)
    out = tuple(torch.zeros((sim.capacity,) + t.shape[1:], dtype=t.dtype, device=DEV) for t in (inst, pos, f))
    return {"case": case, "sim": sim, "in": (inst, pos, f), "out": out}


def _run_step(s):
    case, sim = s["case"], s["sim"]
    if case["pipelined"]:
        sim.set_state(*s["in"], check=False, presorted=case["presorted"])
        sim.step(case["steps"])
        return sim.state_into(s["out"])
    sim.set_state(*s["in"], presorted=case["presorted"])
    sim.step(case["steps"])
    sim.state(out=s["out"])
    return s["out"]


def _dropin_inputs(case, seed):
    """One jittered point per thinning cell (dx / 4): the density the reference's step settles at."""
    g = _generator(seed)
    C, W, cs2 = _lattice("D2Q7")
    x = _grid((4 * case["nx"], 4 * case["ny"]), g, 0.25)
    u = _modes(x, (case["nx"], case["ny"]), g)
    return x, _feq(torch.full((len(x),), 1 / 16, dtype=x.dtype, device=DEV), u, C, W, cs2)


def _prepare_dropin(case, seed):
    pos, f = _in_precision(case, *_dropin_inputs(case, seed))
    sim = GpuSimulator(pos.cpu().numpy(), f.cpu().numpy(), 0.6, precision=case["precision"],
                       box=((0.0, 0.0), (case["nx"], case["ny"])), periodic=True, rho_rest=1 / 16)
    return {"case": case, "sim": sim}


def _run_dropin(s):
    for _ in range(s["case"]["steps"]):
        s["sim"].step()
    return tuple(_rows(a.tensor, 16 * s["case"]["nx"] * s["case"]["ny"]) for a in (s["sim"].pos_m, s["sim"].f_m))


def _prepare_pulse(case, seed):
    h = case["half"]
    rng = np.random.default_rng(seed)
    i, j = np.meshgrid(np.arange(-h, h + 1), np.arange(-h, h + 1), indexing="ij")
    pos = np.stack([i.reshape(-1), j.reshape(-1)], 1) + rng.uniform(-0.05, 0.05, ((2 * h + 1) ** 2, 2))
    rho = np.where((i == 0) & (j == 0), 1.5, 1.0).reshape(-1)
    f = rho[:, None] * np.array([0.5] + [1 / 12] * 6)
    return {"case": case, "in": (pos.astype(np.float32), f.astype(np.float32))}


def _run_pulse(s):
    sim = GpuSimulator(*s["in"], 0.6, precision=s["case"]["precision"])
    for _ in range(s["case"]["steps"]):
        sim.step()
    rows = 16 * (2 * (s["case"]["half"] + s["case"]["steps"] + 1)) ** 2  # what the spread can reach
    return tuple(_rows(a, rows) for a in sim.moments())


def _gradient_inputs(case, seed):
    g = _generator(seed)
    C, W, cs2 = _lattice("D2Q9")
    n = case["n"]
    x = _grid((n, n), g)
    f = _feq(torch.ones(len(x), dtype=x.dtype, device=DEV), _modes(x, (n, n), g), C, W, cs2)
    k = torch.floor(torch.rand((2, 2), generator=g, dtype=x.dtype, device=DEV) * 4) + 1
    return x, f, torch.full((1,), 0.6, dtype=x.dtype, device=DEV), k * (2 * math.pi / n), C


def _loss(pos, f, k, C):
    """Mean square distance of the velocities from a target shear flow."""
    u = (f @ C) / f.sum(1, keepdim=True)
    t = 0.02 * torch.sin(pos.flip(1) * k[0] + k[1])
    return ((u - t) ** 2).sum(1).mean()


def _prepare_gradient(case, seed):
    x, f, tau, k, C = _gradient_inputs(case, seed)
    n = case["n"]
    sim = Simulation([Instance(dims=(n, n), tau=0.6)], lattice="D2Q9", precision=case["precision"], dx=1.0, r_res=1.5,
                     cell=1.0, moment_capacity=4 * n * n)
    return {"case": case, "sim": sim, "tape": Tape(sim), "in": (x, f, tau), "target": (k, C)}


def _run_gradient(s):
    case = s["case"]
    x, f, tau = (t.clone().requires_grad_(True) for t in s["in"])
    _, pos, ft = rollout(s["sim"], None, x, f, tau, case["steps"], case["every"], tape=s["tape"])
    loss = _loss(pos, ft, *s["target"])
    loss.backward()
    return {"loss": loss.detach(), "pos": pos.detach(), "f": ft.detach(), "g_pos": x.grad, "g_f": f.grad,
            "g_tau": tau.grad}


def _lbm_f(case, seed):
    """Deviation-free f (runs, 7, nj, ni) in float64: a shear wave with a small random perturbation."""
    g = _generator(seed)
    C, W, cs2 = _lattice("D2Q7")
    ni, nj, runs = case["ni"], case["nj"], case["runs"]
    j = torch.arange(nj, dtype=torch.float64, device=DEV) * (2 * math.pi / nj)
    ph = torch.rand(runs, generator=g, dtype=torch.float64, device=DEV) * 2 * math.pi
    u = torch.randn((runs, nj, ni, 2), generator=g, dtype=torch.float64, device=DEV) * 1e-3
    u[..., 0] += 0.01 * torch.sin(j[None] + ph[:, None])[:, :, None]
    rho = 1 + 0.01 * torch.randn((runs, nj, ni), generator=g, dtype=torch.float64, device=DEV)
    return _feq(rho, u, C, W, cs2).movedim(-1, 1).contiguous()


def _taus(case):
    return np.linspace(0.55, 1.0, case["runs"]) if case["runs"] > 1 else np.array([0.7])


def _prepare_lbm(case, seed):
    lb = HexLBM(case["ni"], case["nj"], _taus(case), precision=case["precision"])
    f = _lbm_f(case, seed)
    if case["precision"] == "fp32dev":
        f = f - _lattice("D2Q7")[1][:, None, None]
    lb.state.copy_(f)
    return {"case": case, "lbm": lb}


def _run_lbm(s):
    s["lbm"].step(s["case"]["steps"])
    return s["lbm"].state


def _fields_inputs(case, seed):
    g = _generator(seed)
    C, W, cs2 = _lattice(case["lattice"])
    D = C.shape[1]
    x = _grid((case["n"],) * D, g)
    f = _feq(torch.ones(len(x), dtype=x.dtype, device=DEV), _modes(x, (case["n"],) * D, g), C, W, cs2)
    return x, f, np.arange(0.0, case["n"] + case["bin"], case["bin"])


def _prepare_fields(case, seed):
    x, f, edges = _fields_inputs(case, seed)
    return {"case": case, "in": (x, f, edges)}


def _run_fields(s):
    x, f, edges = s["in"]
    if x.shape[1] == 3:
        return dbm_fields.bin_fields3_device(x, f, edges, edges, edges, s["case"]["lattice"])
    return dbm_fields.bin_fields_device(x, f, edges, edges, s["case"]["lattice"])


def _stage_inputs(case, seed):
    g = _generator(seed)
    C, W, cs2 = _lattice("D2Q7")
    n = case["n"]
    x = _grid((n, n), g) - n / 2
    f = _feq(torch.ones(len(x), dtype=x.dtype, device=DEV), _modes(x, (n, n), g), C, W, cs2)
    return x.float(), f.float(), W.float()


def _prepare_stages(case, seed):
    return {"case": case, "in": _stage_inputs(case, seed)}


def _run_stages(s):
    x, f, f_rest = s["in"]
    pos_c, val_c, dir_c = disperse(x, f, 1.0)
    cp, _ = create_control_points(pos_c, 0.25)
    moved = refine_control_points(cp, pos_c, val_c, dir_c, 1.0, 4)
    out_pos, out_f = resample(pos_c, val_c, dir_c, moved, 1.0, f_rest)
    return [_rows(a.tensor, len(val_c)) for a in (pos_c, val_c, dir_c, cp, moved, out_pos, out_f)]


_PREPARE = {"step": _prepare_step, "dropin": _prepare_dropin, "pulse": _prepare_pulse, "gradient": _prepare_gradient,
            "lbm": _prepare_lbm, "fields": _prepare_fields, "stages": _prepare_stages}
_RUN = {"step": _run_step, "dropin": _run_dropin, "pulse": _run_pulse, "gradient": _run_gradient, "lbm": _run_lbm,
        "fields": _run_fields, "stages": _run_stages}


# ---- least work ---------------------------------------------------------------------------------------


def _step_flops(points, Q, D, R, steps):
    """Components within r of a point: Q times the ball's volume in cells (one moment per cell).  Each
    such pair needs its displacement and squared distance (3 D - 1) for the refine, the weight and
    the gather, the refine sums (D + 1 weighted terms), a root and a sum for the weight, and a root,
    a product and a sum for the gather; per component the collision and the exponential."""
    ball = math.pi * R * R if D == 2 else 4 / 3 * math.pi * R ** 3
    return points * steps * (Q * ball * (3 * (3 * D - 1) + 2 * (D + 1) + 3 + 5) + Q * 20)


def work(case):
    kind = case["kind"]
    real = 8 if case.get("precision") == "fp64" else 4
    if kind == "step":
        D = 3 if case["lattice"].startswith("D3") else 2
        Q = int(case["lattice"].split("Q")[1])
        points = sum(math.prod(dims) for dims, _ in _boxes(case))
        row = 4 + (D + Q) * real
        return {"bytes": 2 * points * row * case["steps"], "flops": _step_flops(points, Q, D, _r_res(case), case["steps"])}
    if kind == "dropin":
        points = 16 * case["nx"] * case["ny"]
        return {"bytes": 2 * points * 9 * real * case["steps"], "flops": _step_flops(points, 7, 2, 4.0, case["steps"])}
    if kind == "pulse":
        points = 16 * (2 * case["half"] + case["steps"]) ** 2
        return {"bytes": 2 * points * 9 * real * case["steps"], "flops": _step_flops(points, 7, 2, 4.0, case["steps"])}
    if kind == "gradient":  # forward, recomputation, and two products per forward operation
        points = case["n"] ** 2
        return {"bytes": 8 * points * 11 * real * case["steps"],
                "flops": 4 * _step_flops(points, 9, 2, 1.5, case["steps"])}
    if kind == "lbm":
        nodes = case["ni"] * case["nj"] * case["runs"] * case["steps"]
        return {"bytes": nodes * 14 * real, "flops": nodes * 90}
    if kind == "fields":
        D = 3 if case["lattice"].startswith("D3") else 2
        Q = int(case["lattice"].split("Q")[1])
        points, bins = case["n"] ** D, math.ceil(case["n"] / case["bin"]) ** D
        return {"bytes": points * (Q + D) * 8 + bins * (1 + D) * 8, "flops": points * Q * (1 + 2 * D)}
    nc = 7 * case["n"] ** 2
    cps = min(nc, 16 * case["n"] ** 2)
    return {"bytes": case["n"] ** 2 * 36 + nc * 16 * 4 + cps * (4 * 8 + 28), "flops": cps * 7 * math.pi * 60}


# ---- 64-bit statement of the method ---------------------------------------------------------------------


class _Box:
    """One periodic box of cells and its moments: cell index, offset in the cell, f."""

    def __init__(self, dims, tau, cell, off, f):
        self.dims, self.tau, self.cell, self.off, self.f = dims, tau, cell, off, f


def _index(dims, c):
    n = torch.tensor(dims, device=DEV)
    c = torch.remainder(c, n)
    i = c[:, -1]
    for a in range(len(dims) - 2, -1, -1):
        i = i * dims[a] + c[:, a]
    return i


def _coords(dims, cell):
    out = []
    for n in dims:
        out.append(cell % n)
        cell = cell // n
    return torch.stack(out, 1)


def _load(dims, tau, x, f, cell_size):
    s = x / cell_size
    c = torch.floor(s)
    key = _index(dims, c.long())
    order = torch.argsort(key, stable=True)
    return _Box(dims, tau, key[order], (s - c)[order], f[order]), order


def _table(ncells, cell):
    """Items of every cell, one column per item: index or -1 (cells sorted)."""
    n = torch.bincount(cell, minlength=ncells)
    start = torch.cumsum(n, 0) - n
    slots = max(int(n.max()), 1)
    s = torch.arange(slots, device=DEV)[None]
    return torch.where(s < n[:, None], start[:, None] + s, -1)


def _pairs(dims, ref_cell, ref_off, table, off, cd, R):
    """Candidate items of every reference point within R for displacement cd: (item, inside, e)."""
    c0 = _coords(dims, ref_cell)
    spans = [range(math.floor(-float(v) - R), math.floor(1 - float(v) + R) + 1) for v in cd]
    for o in itertools.product(*spans):
        shift = torch.tensor(o, device=DEV)
        cells = _index(dims, c0 + shift)
        for s in range(table.shape[1]):
            item = table[cells, s]
            ok = item >= 0
            if not bool(ok.any()):
                continue
            item = item.clamp(min=0)
            e = off[item] + (shift + cd - ref_off)
            yield item, ok & ((e * e).sum(1) <= R * R), e


def _distance(e):
    d2 = (e * e).sum(1)
    zero = d2 == 0
    return torch.where(zero, 0.0, torch.sqrt(torch.where(zero, 1.0, d2)))


def _step64(b, C, W, cs2, R, dx_cells, kappa_hard=4, eps=1e-6, rho_rest=1.0):
    """One step of a periodic box: collide, disperse, thin, refine, resample, fill gaps."""
    Q, D = C.shape
    ncells = math.prod(b.dims)
    M = len(b.cell)
    rho = b.f.sum(1)
    feq = _feq(rho, (b.f @ C) / rho[:, None], C, W, cs2)
    f = b.f + (feq - b.f) / b.tau
    # thinning: centroid of the components of each cell
    cd = C * dx_cells
    base = _coords(b.dims, b.cell)
    key, rel = [], []
    for k in range(Q):
        t = b.off + cd[k]
        fl = torch.floor(t)
        key.append(_index(b.dims, base + fl.detach().long()))
        rel.append(t - fl.detach())
    key, rel = torch.cat(key), torch.cat(rel)
    count = torch.bincount(key, minlength=ncells)
    total = torch.zeros((ncells, D), dtype=rel.dtype, device=DEV).index_add(0, key, rel)
    thin = torch.nonzero(count).reshape(-1)
    cen = total[thin] / count[thin][:, None]
    # refine: points that see more than kappa_hard directions move to the exp(f)-weighted centroid
    table = _table(ncells, b.cell)
    kappa = torch.zeros(len(thin), dtype=torch.int64, device=DEV)
    sw = torch.zeros(len(thin), dtype=rel.dtype, device=DEV)
    sx = torch.zeros_like(cen)
    for k in range(Q):
        seen = torch.zeros(len(thin), dtype=torch.bool, device=DEV)
        wk = torch.exp(f[:, k])
        for item, inside, e in _pairs(b.dims, thin, cen.detach(), table, b.off.detach(), cd[k], R):
            seen = seen | inside
            w = torch.where(inside, wk[item], 0.0)
            if cen.requires_grad:  # the same displacement, as a function of the moving ends
                e = e + (b.off[item] - b.off[item].detach()) - (cen - cen.detach())
            sw = sw + w
            sx = sx + w[:, None] * e
        kappa += seen
    p = torch.where((kappa > kappa_hard)[:, None], cen + sx / torch.where(sw > 0, sw, 1.0)[:, None], cen)
    fl = torch.floor(p.detach())
    cell = _index(b.dims, _coords(b.dims, thin) + fl.long())
    order = torch.argsort(cell, stable=True)
    cell, off = cell[order], (p - fl)[order]
    # resample: component weights, then sums per control point and direction
    P = len(cell)
    out = []
    for k in range(Q):
        hits = lambda: _pairs(b.dims, cell, off, table, b.off, cd[k], R)  # noqa: E731
        tot = torch.zeros(M, dtype=rel.dtype, device=DEV)
        for item, inside, e in hits():
            tot = tot.index_add(0, item, torch.where(inside, R - _distance(e), 0.0))
        share = torch.where(tot > 0, f[:, k] / torch.where(tot > 0, tot, 1.0), 0.0)
        acc = torch.zeros(P, dtype=rel.dtype, device=DEV)
        for item, inside, e in hits():
            acc = acc + torch.where(inside, (R - _distance(e)) * share[item], 0.0)
        out.append(acc)
    F = torch.stack(out, 1)
    empty = F < eps
    if bool(empty.any()):
        cps = _table(ncells, cell)
        near = torch.zeros_like(F)
        for item, inside, e in _pairs(b.dims, cell, off, cps, off, torch.zeros_like(cd[0]), R):
            w = torch.where(inside, R - _distance(e), 0.0)
            near = near + w[:, None] * empty[item]
        fill = R / torch.where(near > 0, near, 1.0) * (rho_rest * W)
        F = torch.where(empty & (near > 0), fill, F)
    return _Box(b.dims, b.tau, cell, off, F)


def exact(case, seed):
    if case["kind"] == "step":
        boxes = _boxes(case)
        points = sum(math.prod(dims) for dims, _ in boxes) * case["steps"]
        if case["obstacle"] or case["soft"] or len(boxes) > 40 or points > 4e6:
            return None
        inst, pos, f = _step_inputs(case, seed)
        C, W, cs2 = _lattice(case["lattice"])
        out_i, out_x, out_f = [], [], []
        for i, (dims, tau) in enumerate(boxes):
            b, _ = _load(dims, tau, pos[inst == i], f[inst == i], 1.0)
            for _ in range(case["steps"]):
                b = _step64(b, C, W, cs2, _r_res(case), 1.0)
            out_i.append(torch.full((len(b.cell),), i, dtype=torch.int32, device=DEV))
            out_x.append(_coords(dims, b.cell) + b.off)
            out_f.append(b.f)
        rows = sum(math.prod(dims) for dims, _ in boxes)
        return (torch.nn.functional.pad(torch.cat(out_i), (0, rows - len(torch.cat(out_i)))),
                _rows(torch.cat(out_x), rows), _rows(torch.cat(out_f), rows))
    if case["kind"] == "dropin":
        if case["nx"] * case["ny"] * case["steps"] > 2e4:
            return None
        x, f = _dropin_inputs(case, seed)
        C, W, cs2 = _lattice("D2Q7")
        b, _ = _load((4 * case["nx"], 4 * case["ny"]), 0.6, x, f, 0.25)
        for _ in range(case["steps"]):
            b = _step64(b, C, W, cs2, 4.0, 4.0, rho_rest=1 / 16)
        rows = math.prod(b.dims)
        return _rows((_coords(b.dims, b.cell) + b.off) * 0.25, rows), _rows(b.f, rows)
    if case["kind"] == "gradient":
        if case["n"] ** 2 * case["steps"] > 2e4:
            return None
        x, f, tau, k, C = _gradient_inputs(case, seed)
        W, cs2 = _lattice("D2Q9")[1:]
        x, f, tau = (t.requires_grad_(True) for t in (x, f, tau))
        b, _ = _load((case["n"],) * 2, tau, x, f, 1.0)
        for _ in range(case["steps"]):
            b = _step64(b, C, W, cs2, 1.5, 1.0)
        pos = _coords(b.dims, b.cell) + b.off
        loss = _loss(pos, b.f, k, C)
        loss.backward()
        return {"loss": loss.detach(), "pos": pos.detach(), "f": b.f.detach(), "g_pos": x.grad, "g_f": f.grad,
                "g_tau": tau.grad}
    if case["kind"] == "lbm":
        C, W, cs2 = _lattice("D2Q7")
        f = _lbm_f(case, seed)
        tau = torch.tensor(_taus(case), device=DEV)[:, None, None, None]
        for _ in range(case["steps"]):
            g = f.movedim(1, -1)
            rho = g.sum(-1)
            g = g + (_feq(rho, (g @ C) / rho[..., None], C, W, cs2) - g) / tau
            hop = [(0, 0), (1, 0), (0, 1), (-1, 1), (-1, 0), (0, -1), (1, -1)]
            f = torch.stack([torch.roll(g[..., k], (dj, di), (1, 2)) for k, (di, dj) in enumerate(hop)], 1)
        return f - W[:, None, None] if case["precision"] == "fp32dev" else f
    if case["kind"] == "fields":
        x, f, edges = _fields_inputs(case, seed)
        C = _lattice(case["lattice"])[0]
        e = torch.tensor(edges, device=DEV)
        n = len(edges) - 1
        D = C.shape[1]
        b = (torch.searchsorted(e, x.contiguous(), right=True) - 1).clamp(max=n - 1)
        key = b[:, D - 1]
        for a in range(D - 2, -1, -1):
            key = key * n + b[:, a]
        parts = [f.sum(1)] + [(f * C[:, a]).sum(1) for a in range(D)]
        return [torch.zeros(n ** D, dtype=f.dtype, device=DEV).index_add(0, key, v).reshape((n,) * D) for v in parts]
    if case["kind"] == "stages":
        x, f, _ = _stage_inputs(case, seed)
        C = _lattice("D2Q7")[0]
        pos = (x.double()[:, None, :] + C).reshape(-1, 2)
        return [pos, f.double().reshape(-1), None, None, None, None, None]
    return None
