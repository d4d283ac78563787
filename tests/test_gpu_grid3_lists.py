"""The brick lists of the 3D grid kernels belong to creation and to a change of obstacle: a first step, and a
step after a new inflow velocity, allocate nothing and wait for nothing, so a captured stream takes them."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = (26, 24, 24)


def _sim(**extra):
    from direbm_gb300.lattices import D3Q19
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    rng = np.random.default_rng(3)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in DIMS], indexing="ij"), -1).reshape(-1, 3)
    x = c + rng.uniform(0.2, 0.8, c.shape)
    if "obstacle" in extra:
        center, radius = extra["obstacle"]
        x = x[((x - np.asarray(center)) ** 2).sum(1) > (radius + 0.5) ** 2]
    u = np.zeros_like(x)
    u[:, 0] = 0.03
    sim = Simulation([Instance(dims=DIMS, tau=0.7, inflow=((0.03, 0.0, 0.0), 2), **extra)], lattice="D3Q19",
                     precision="fp32dev", dx=1.0, r_res=1.5, cell=1.0, graphs=False)
    sim.set_state(None, x, equilibrium(np.ones(len(x)), u, D3Q19))
    return sim


@pytest.mark.parametrize("obstacle", [False, True])
def test_steps_under_capture(obstacle):
    extra = {"obstacle": ((13.0, 12.0, 12.0), 2.0)} if obstacle else {}
    sims = [_sim(**extra) for _ in range(2)]
    held = sims[0].device_bytes
    for velocity in (0.03, 0.05):  # the very first steps, then those after a new inflow
        for sim in sims:
            sim.set_inflow(0, (velocity, 0.0, 0.0), 2)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            sims[0].step(2)
        g.replay()
        torch.cuda.synchronize()
        sims[1].step(2)
        for a, b in zip(sims[0].state_numpy(), sims[1].state_numpy()):
            np.testing.assert_array_equal(a, b)
    assert sims[0].device_bytes == held


def test_obstacle_moved_between_steps():
    """New lists in the old buffers: the bits are those of the untiled kernels."""
    outs = []
    for grid in (True, False):
        sim = _sim(obstacle=((12.0, 12.0, 12.0), 2.0))
        sim.set_dense_stencil(grid)
        sim.step(2)
        sim.set_obstacle(0, (14.0, 12.0, 12.0), 1.5)
        sim.step(2)
        sim.set_obstacle(0, (0.0, 0.0, 0.0), 0.0)
        sim.step(2)
        outs.append(sim.state_numpy())
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
