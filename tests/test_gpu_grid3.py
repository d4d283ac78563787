"""The 3D grid window kernels against the untiled ones: every bit has to agree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,r_res", [("D3Q19", 1.5), ("D3Q19", 1.2), ("D3Q13", 1.5), ("D3Q13", 1.05)])
@pytest.mark.parametrize("case", ["jittered", "borders", "crowded", "very_crowded", "sparse", "negative_rho",
                                  "infinite_f", "bounded", "obstacle", "late"])
def test_grid3_equals_untiled(case, lattice, r_res):
    """borders: offsets at and around cell borders (wider windows); crowded, very_crowded: cells with
    several moments, up to and beyond the list; obstacle: bricks left to the untiled kernels beside
    clear ones; late: a longer run, over which some cells come to hold two moments."""
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    lat = get(lattice)
    dims = (58, 37, 40) if case == "obstacle" else (21, 18, 26)
    rng = np.random.default_rng(5)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    off = rng.uniform(0.1, 0.9, c.shape)
    if case == "borders":
        off[::3] = rng.choice([0.0, 1e-7, 5e-5, 0.5, 0.50003, float(np.float32(1) - np.float32(2.0 ** -24))], off[::3].shape)
    if case in ("crowded", "very_crowded"):
        more = rng.integers(0, len(c), len(c) // (100 if case == "crowded" else 3))
        more = np.concatenate([more, np.repeat(more[:3], 3)])
        c = np.concatenate([c, c[more]])
        off = np.concatenate([off, rng.uniform(0, 1, (len(more), 3))])
    if case == "sparse":
        c, off = c[::11], off[::11]
    extra = {}
    if case == "bounded":
        inside = ((c >= 6) & (c < np.array(dims) - 6)).all(1)
        c, off = c[inside], off[inside]
    if case == "obstacle":
        extra = {"obstacle": ((16.0, 18.0, 20.0), 6.0), "inflow": ((0.04, 0.0, 0.0), 2)}
        keep = ((c + off - [16.0, 18.0, 20.0]) ** 2).sum(1) > 6.5 ** 2
        c, off = c[keep], off[keep]
    x = c + off
    u = 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 2]), np.sin(x[:, 0])], 1)
    f = equilibrium(np.ones(len(x)), u, lat)
    if case == "negative_rho":
        f[len(f) // 2] *= -0.5
    if case == "infinite_f":
        f[len(f) // 2, 3] = np.inf
    steps = {"infinite_f": 1, "bounded": 1, "late": 20}.get(case, 3)
    outs = []
    for grid in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7, periodic=case != "bounded", **extra)], lattice=lattice,
                         precision="fp32dev", dx=1.0, r_res=r_res, cell=1.0, moment_capacity=2 * len(x))
        sim.set_dense_stencil(grid)
        sim.set_state(None, x, f)
        sim.step(steps)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
