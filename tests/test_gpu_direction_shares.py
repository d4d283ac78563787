"""Blocks that share a tile's directions (small boxes), and the sizes at which they stop, against the
row-segment kernels: every bit has to agree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fill", ["full", "corner", "crowded"])
@pytest.mark.parametrize("dims", [(31, 33), (130, 141), (230, 240), (330, 320), (905, 801)])
@pytest.mark.parametrize("lattice,cell,r_res", [("D2Q7", 0.25, 1.0), ("D2Q7", 1.0, 1.5), ("D2Q9", 1.0, 1.5)])
def test_shared_directions_equal_row_segments(lattice, cell, r_res, dims, fill):
    """full: the shares fall from one direction a block to none with the size; corner: a large box that is
    mostly empty (few moments: shared; empty tiles); crowded: tiles left to the fallback and empty
    directions beside holes."""
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    lat = get(lattice)
    rng = np.random.default_rng(17)
    c = np.stack(np.meshgrid(np.arange(dims[0]), np.arange(dims[1])), -1).reshape(-1, 2).astype(np.float64)
    if fill == "corner":
        c = c[(c < 29).all(1)]
    off = rng.uniform(0.05, 0.95, c.shape)
    if fill == "crowded":
        hole = ((c >= 8) & (c < 20)).all(1)
        c, off = c[~hole], off[~hole]
        more = np.repeat(c[:40:8], 9, axis=0)
        c, off = np.concatenate([c, more]), np.concatenate([off, rng.uniform(0, 1, more.shape)])
    x = (c + off) * cell
    u = 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 0])], 1)
    f = equilibrium(np.full(len(x), cell * cell), u, lat)
    outs = []
    for fast in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7, periodic=True, rho_rest=cell * cell)], lattice=lattice,
                         precision="fp32dev", dx=1.0, r_res=r_res, cell=cell, moment_capacity=2 * int(np.prod(dims)))
        sim.set_dense_stencil(fast)
        sim.set_state(None, x, f)
        sim.step(2)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
