"""The grid window kernels (displacements that are not whole cells, or R = 4 cells) against the
row-segment kernels: the same hits in the same order, so every bit has to agree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 32, 128])
@pytest.mark.parametrize("lattice,cell,r_res", [("D2Q7", 0.25, 1.0), ("D2Q7", 1.0, 1.5), ("D2Q7", 1.0, 1.1),
                                                ("D2Q9", 0.25, 1.0), ("D2Q9", 0.25, 0.9)])
@pytest.mark.parametrize("case", ["jittered", "borders", "crowded", "very_crowded", "sparse", "negative_rho",
                                  "infinite_f", "bounded"])
def test_grid_windows_equal_row_segments(case, lattice, cell, r_res, width):
    """borders: offsets at and around cell borders, where a window is one cell wider; crowded: cells with
    two to five moments (the ordered list); very_crowded: more than the list takes (fallback); sparse:
    mostly empty cells; negative_rho, infinite_f: not for the gather's sums; bounded: a box with walls."""
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    lat = get(lattice)
    n0, n1 = 45, 38  # cells; ragged against every tile shape
    rng = np.random.default_rng(11)
    c = np.stack(np.meshgrid(np.arange(n0), np.arange(n1)), -1).reshape(-1, 2).astype(np.float64)
    off = rng.uniform(0.05, 0.95, c.shape)
    if case == "borders":
        off[::3] = rng.choice([0.0, 1e-7, 5e-5, 1 - 5e-5, float(np.float32(1) - np.float32(2.0 ** -24))], off[::3].shape)
    if case in ("crowded", "very_crowded"):
        more = rng.integers(0, len(c), len(c) // (40 if case == "crowded" else 2))
        more = np.concatenate([more, np.repeat(more[:3], 3)])
        c = np.concatenate([c, c[more]])
        off = np.concatenate([off, rng.uniform(0, 1, (len(more), 2))])
    if case == "sparse":
        c, off = c[::17], off[::17]
    if case == "bounded":
        inside = ((c >= 14) & (c < np.array([n0, n1]) - 14)).all(1)
        c, off = c[inside], off[inside]
    x = (c + off) * cell
    u = 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 0])], 1)
    f = equilibrium(np.full(len(x), cell * cell), u, lat)
    if case == "negative_rho":
        f[len(f) // 2] *= -0.5
    if case == "infinite_f":
        f[len(f) // 2, 3] = np.inf
    steps = 1 if case in ("infinite_f", "bounded") else 3
    outs = []
    for grid in (True, False):
        sim = Simulation([Instance(dims=(n0, n1), tau=0.7, periodic=case != "bounded", rho_rest=cell * cell)],
                         lattice=lattice, precision="fp32dev", dx=1.0, r_res=r_res, cell=cell, moment_capacity=2 * len(x))
        sim.set_tiling(width, False)
        sim.set_dense_stencil(grid)
        sim.set_state(None, x, f)
        sim.step(steps)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
