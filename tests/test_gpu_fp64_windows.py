"""FP64 window sums (candidates by FP32, hits in FP64) against the dense-grid oracle: the decisions agree
exactly (moment count, and with them every position), the values to the FP64 tolerance of the other stage
tests, 1e-12 of the largest."""

import numpy as np
import pytest

from oracle import grid_step

pytestmark = pytest.mark.gpu

CASES = {
    # lattice, dims, dx, r_res, cell, periodic, obstacle
    "crowded": ("D2Q9", (19, 13), 1.0, 1.5, 1.0, True, None),  # windows beyond a thread's list
    "quarter_cells": ("D2Q7", (41, 37), 1.0, 1.0, 0.25, True, None),
    "wide": ("D2Q9", (45, 46), 1.0, 9.0, 1.0, True, None),  # displacements beyond the block's table
    "far": ("D2Q9", (12, 3040), 3000.0, 1.5, 1.0, False, None),  # displacements of thousands of cells
    "ragged_far": ("D2Q7", (12, 3040), 3333.3, 1.5, 1.0, False, None),
    "bounded": ("D2Q7", (17, 23), 1.0, 1.5, 1.0, False, None),
    "borders": ("D2Q9", (21, 15), 1.0, 1.5, 1.0, True, None),  # offsets and distances at the bounds
    "disc": ("D2Q9", (30, 33), 1.0, 1.5, 1.0, True, ((15.0, 16.0), 4.0)),
    "box": ("D3Q19", (11, 10, 12), 1.0, 1.5, 1.0, True, None),
    "crowded_box": ("D3Q19", (10, 11, 10), 1.0, 1.2, 1.0, True, None),
    "sphere": ("D3Q13", (17, 16, 16), 1.0, 1.2, 1.0, True, ((8.0, 8.5, 8.0), 2.5)),
}


@pytest.mark.parametrize("case", list(CASES))
def test_fp64_windows_match_oracle(case):
    from direbm_gb300.sim import Instance, Simulation
    from oracle.lattices import BY_NAME
    from oracle.physics import equilibrium

    lattice, dims, dx, r_res, cell, periodic, obstacle = CASES[case]
    lat = BY_NAME[lattice]
    D = len(dims)
    rng = np.random.default_rng(3)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, D).astype(np.float64)
    off = rng.uniform(0.05, 0.95, c.shape)
    if case.endswith("far"):
        keep = (c[:, 1] < 40) | (c[:, 1] >= 3000)
        c, off = c[keep], off[keep]
    if case == "bounded":
        keep = ((c >= 4) & (c < np.array(dims) - 4)).all(1)
        c, off = c[keep], off[keep]
    if case == "wide":
        c, off = c[::3], off[::3]
    if case == "borders":
        off = rng.choice([0.0, 2.0 ** -40, 0.25, 0.5, 0.75, 1 - 2.0 ** -30], c.shape)
    if case.startswith("crowded"):
        more = np.repeat(c[[7, len(c) // 2, -3]], 130, axis=0)
        c = np.concatenate([c, more])
        off = np.concatenate([off, rng.uniform(0, 1, more.shape)])
    x = (c + off) * cell
    if obstacle:
        keep = ((x - np.array(obstacle[0])) ** 2).sum(1) > (obstacle[1] + 0.2) ** 2
        x = x[keep]
    u = 0.03 * np.sin(x + np.arange(D)) * np.cos(x[:, ::-1])
    f = equilibrium(np.full(len(x), cell ** D), u, lat)
    kw = dict(dims=dims, periodic=periodic, tau=0.7, rho_rest=cell ** D, obstacle=obstacle)
    spec = grid_step.GridSpec(lattice=lat, dx=dx, r_res=r_res, cell=cell, kappa_hard=4,
                              instances=[grid_step.Instance(**kw)])
    st = grid_step.from_world(spec, np.zeros(len(x), np.int64), x, f)
    sim = Simulation([Instance(**kw)], lattice=lattice, precision="fp64", dx=dx, r_res=r_res, cell=cell,
                     moment_capacity=2 * len(x))
    sim.set_state(None, x, f)
    for _ in range(1 if case == "borders" else 2):  # borders: ties only in the first step
        st = grid_step.step(spec, st)
        sim.step(1)
        _, xo, fo = grid_step.to_world(spec, st)
        _, xg, fg = sim.state_numpy()
        assert len(xg) == len(xo) > 0
        np.testing.assert_allclose(xg, xo, rtol=0, atol=1e-12 * max(dims) * cell)
        np.testing.assert_allclose(fg, fo, rtol=0, atol=1e-12 * np.abs(fo).max())
    sim.close()
