"""Simulators of different shared-memory needs side by side: what one sets up for its kernels may not take away
what another's launches need."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [("D2Q7", 4.0, 4.0, (40, 44)), ("D2Q7", 2.5, 3.6, (40, 44)), ("D2Q7", 1.0, 1.5, (40, 44)),
          ("D2Q7", 1.0, 1.02, (40, 44)), ("D2Q9", 1.0, 1.5, (40, 44)), ("D2Q9", 1.0, 0.5, (40, 44)),
          ("D2Q9", 3.0, 1.9, (40, 44)), ("D2Q9", 1.25, 1.5, (40, 44)), ("D2Q9", 1.25, 4.0, (40, 44))]


def _sim(lattice, dx, r_res, dims, width):
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    rng = np.random.default_rng(1)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, 2)
    x = c + rng.uniform(0.2, 0.8, c.shape)
    sim = Simulation([Instance(dims=dims, tau=0.7)], lattice=lattice, precision="fp32dev", dx=dx, r_res=r_res, cell=1.0)
    sim.set_tiling(width, False)
    sim.set_state(None, x, equilibrium(np.ones(len(x)), 0.02 * np.sin(x), get(lattice)))
    return sim


@pytest.mark.parametrize("graphs_first", [False, True])
def test_side_by_side(graphs_first):
    alone = []
    for shape in SHAPES:
        sim = _sim(*shape, 32)
        sim.step(3)
        alone.append(sim.state_numpy())
        sim.close()
    sims = [_sim(*shape, 32) for shape in SHAPES]
    if graphs_first:
        for sim in sims:
            sim.step(1)
    small = [_sim(*shape, 8 if i % 2 else 64) for i, shape in enumerate(SHAPES[::-1])]  # other needs, created later
    for sim, ref in zip(sims, alone):
        sim.step(2 if graphs_first else 3)
        for a, b in zip(sim.state_numpy(), ref):
            np.testing.assert_array_equal(a, b)
    for sim in sims + small:
        sim.close()
