"""Dense kernels of whole-cell displacements other than one cell, and of radii whose windows do not fit four
cells: each against the row-segment kernels, every bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# widths of a window: 2 and 3 cells (R <= 1), 4 (R <= 1.5), 5; radii at the lines between them
@pytest.mark.parametrize("dx,r_res", [(1.0, 0.4), (1.0, 0.7), (1.0, 0.9999), (2.0, 0.9), (2.0, 1.0), (2.0, 1.4999),
                                      (2.0, 1.5), (2.0, 1.99), (3.0, 1.2), (1.0, 1.56), (1.0, 1.7), (1.0, 1.99)])
@pytest.mark.parametrize("width", [8, 32, 128])
def test_far_dense_equals_row_segments(dx, r_res, width):
    from direbm_gb300.sim import Instance, Simulation
    from oracle.lattices import D2Q9
    from oracle.physics import equilibrium

    dims = (37, 29)
    rng = np.random.default_rng(9)
    c = np.stack(np.meshgrid(np.arange(dims[0]), np.arange(dims[1]), indexing="ij"), -1).reshape(-1, 2).astype(float)
    off = rng.uniform(0, 1, c.shape)
    off[::6] = rng.choice([0.0, 1e-7, 5e-5, 0.5, 0.50003, float(np.float32(1) - np.float32(2.0 ** -24))], off[::6].shape)
    second = rng.integers(0, len(c), 20)
    x = np.concatenate([c + off, c[second] + rng.uniform(0, 1, (20, 2))])
    u = 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 0])], 1)
    f = equilibrium(np.ones(len(x)), u, D2Q9)
    outs = []
    for dense in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7)], lattice="D2Q9", precision="fp32dev", dx=dx, r_res=r_res,
                         cell=1.0, moment_capacity=2 * len(x))
        sim.set_tiling(width, False)
        sim.set_dense_stencil(dense)
        sim.set_state(None, x, f)
        sim.step(2)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
