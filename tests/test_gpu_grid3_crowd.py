"""3D grid kernels where bricks are left to the untiled code: one dense spot, a state crowded all over, and few
bricks whose directions are shared by blocks.  Every bit against the untiled kernels."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice", ["D3Q19", "D3Q13"])
@pytest.mark.parametrize("dims", [(21, 18, 26), (64, 48, 40)])  # directions shared, and a block per brick
@pytest.mark.parametrize("case", ["regular", "spot", "corner", "crowded", "spot_and_obstacle"])
def test_deferred_bricks(lattice, dims, case):
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    rng = np.random.default_rng(12)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    extra = {}
    if case.startswith("spot"):  # more further items than a brick's list takes, in 1 of 64 cells of the box
        box = np.array([8, 8, 8]) if dims[0] > 32 else np.array([5, 5, 5])
        spot = c[(c < box).all(1)]
        c = np.concatenate([c] + [spot] * (2 if dims[0] < 32 else 1))
    if case == "corner":
        c = c[(c < np.array(dims) * 0.35).all(1)]
    if case == "crowded":
        c = np.concatenate([c, c[rng.integers(0, len(c), len(c) // 10)]])
    x = c + rng.uniform(0.05, 0.95, c.shape)
    if case == "spot_and_obstacle":
        if dims[0] < 32:
            pytest.skip("a sphere needs more room in a periodic box")
        extra = {"obstacle": ((44.0, 24.0, 20.0), 3.0)}
        x = x[((x - [44.0, 24.0, 20.0]) ** 2).sum(1) > 3.5 ** 2]
    u = 0.02 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 2]), np.sin(x[:, 0])], 1)
    f = equilibrium(np.ones(len(x)), u, get(lattice))
    bricks = int(np.prod([-(-n // 8) for n in dims]))
    outs = []
    for grid in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7, **extra)], lattice=lattice, precision="fp32dev", dx=1.0,
                         r_res=1.5, cell=1.0, moment_capacity=len(x) + int(np.prod(dims)))
        sim.set_dense_stencil(grid)
        sim.set_state(None, x, f)
        sim.step(1)
        deferred = sim.trace("deferred").cpu().numpy().view(np.uint32)
        if grid and case == "regular":
            assert (deferred == 0).all()
        elif grid and case == "crowded":
            assert (deferred == bricks).all()
        elif grid and case.startswith("spot"):
            assert 0 < deferred[0] < bricks and 0 < deferred[2] < bricks
        sim.step(2)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
