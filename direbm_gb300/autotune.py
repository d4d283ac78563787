"""Autotuner for the launch configuration of the window kernels.

Which setting acts depends on the kernels that serve the box (``Simulation.window_path``):

- "tiles" (2D FP32): one 256-thread block per tile of w x 256/w cells stages the tile plus a halo in
  shared memory; the halo share of the staged region, the staging capacity and the row-segment lengths
  all depend on w, and the kernels can be launched one block per tile or persistently (a few resident
  blocks per SM striding over the tile list).  ``CANDIDATES``: (w, persistent).
- "bricks" (FP64, obstacles in 2D, the soft spawn, 3D without the grid kernels): each block takes a brick of
  256 cells; its width along x is the choice (``BRICK_CANDIDATES`` in 3D, ``BRICK_CANDIDATES_2D``).
- "grid3" (the 3D grid kernels): nothing to choose.

Every setting gives bit-identical results, so the choice is purely a speed question:
``autotune`` times a short run of the simulator's own step from one snapshot for each candidate
and keeps the fastest.  Choices are cached in a JSON file keyed by the GPU, the lattice, the
precision, the kernels, the radius and displacement in cell units and the moment density, so a later
run with the same shape of problem skips the timing.
"""

from __future__ import annotations

import json
import os
from pathlib import Path

import torch

from .sim import Simulation

CANDIDATES = tuple((w, p) for w in (32, 16, 64, 8) for p in (False, True))
BRICK_CANDIDATES = (8, 4, 16, 32)  # 3D brick widths along x (8 x 8 x 4, 4 x 8 x 8, 16 x 4 x 4, 32 x 4 x 2)
BRICK_CANDIDATES_2D = (16, 8, 32, 64)


def cache_file() -> Path:
    p = os.environ.get("DIREBM_GB300_TUNE_CACHE")
    return Path(p) if p else Path.home() / ".cache" / "direbm_gb300" / "tiling.json"


def problem_key(sim: Simulation, moments: int) -> str:
    dev = torch.cuda.get_device_name(sim.device)
    density = moments / max(sim.ncells, 1)
    return (f"{dev}|{sim.lattice.name}|{sim.precision}|{sim.window_path()}|R={sim.r_res / sim.cell:.4g}|cd={sim.dx / sim.cell:.4g}"
            f"|density={density:.2g}")


def _load(path: Path) -> dict:
    try:
        return json.loads(path.read_text())
    except (OSError, ValueError):
        return {}


def apply_cached(sim: Simulation) -> dict | None:
    """Apply a cached choice for this problem, if there is one; returns it."""
    entry = _load(cache_file()).get(problem_key(sim, sim.count()))
    if entry:
        if entry.get("brick_width"):
            sim.set_brick_width(entry["brick_width"])
        else:
            sim.set_tiling(entry["tile_width"], entry["persistent"])
    return entry


def _times(sim: Simulation, candidates, apply, steps: int) -> list:
    """Milliseconds per step of the loaded state under each candidate; the state is left as it was."""
    snap = sim.snapshot()
    it = sim.iteration
    out = []
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.device(sim.device):
        for c in candidates:
            apply(c)
            sim.restore(snap)
            sim.step(1)  # warm-up: captures this configuration's graphs
            sim.restore(snap)
            torch.cuda.synchronize()
            e0.record()
            sim.step(steps)
            e1.record()
            torch.cuda.synchronize()
            out.append(e0.elapsed_time(e1) / steps)
    best = min(zip(out, range(len(out))))[1]
    apply(candidates[best])
    sim.restore(snap, it)
    return out


def _store(key: str, entry: dict) -> None:
    path = cache_file()
    data = _load(path)
    data[key] = entry
    try:
        path.parent.mkdir(parents=True, exist_ok=True)
        path.write_text(json.dumps(data, indent=1, sort_keys=True))
    except OSError:
        pass


def autotune(sim: Simulation, steps: int = 2, candidates=CANDIDATES, use_cache: bool = True) -> dict:
    """Time ``steps`` steps of the loaded state under each candidate of the setting that acts on this machine
    (``candidates``: the (tile width, persistent) ones), apply the fastest and return {tile_width,
    persistent, brick_width, ms_per_step, timings, path}; what does not act keeps its value.  The
    simulator's state and iteration count are left as they were."""
    moments = sim.count()
    key = problem_key(sim, moments)
    if use_cache:
        hit = apply_cached(sim)
        if hit:
            return dict(hit, cached=True)
    path = sim.window_path()
    if path == "tiles":
        ms = _times(sim, candidates, lambda c: sim.set_tiling(*c), steps)
        timings = {f"{w}x{256 // w}{'-persistent' if p else ''}": t for (w, p), t in zip(candidates, ms)}
    else:
        if path == "grid3":
            widths = (sim.brick_width(),)
        else:
            widths = BRICK_CANDIDATES if sim.lattice.D == 3 else BRICK_CANDIDATES_2D
        ms = _times(sim, widths, sim.set_brick_width, steps)
        timings = {f"brick{w}" if path == "bricks" else path: t for w, t in zip(widths, ms)}
    w, pers = sim.tiling() if sim.lattice.D == 2 else (None, None)
    entry = {"tile_width": w, "persistent": pers, "ms_per_step": float(min(ms)), "timings": timings, "path": path}
    if path != "tiles":
        entry["brick_width"] = sim.brick_width()
    if use_cache:
        _store(key, entry)
    return dict(entry, cached=False)
