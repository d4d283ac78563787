"""A negative density, or an f that is not finite, takes its own instance's gather off the dense and grid
kernels, not the whole batch's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,r_res,dims", [("D2Q9", 1.5, (40, 36)), ("D2Q7", 1.5, (40, 36)),
                                                ("D3Q19", 1.5, (16, 16, 16))])
@pytest.mark.parametrize("odd", ["negative_rho", "infinite_f"])
def test_one_odd_instance(lattice, r_res, dims, odd):
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    rng = np.random.default_rng(8)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, len(dims)).astype(float)
    x = c + rng.uniform(0.2, 0.8, c.shape)
    u = 0.02 * np.sin(x)
    f = equilibrium(np.ones(len(x)), u, get(lattice))
    members = 3
    inst = np.repeat(np.arange(members), len(x))
    X, F = np.tile(x, (members, 1)), np.tile(f, (members, 1))
    pick = len(x) + len(x) // 2  # in the second instance
    if odd == "negative_rho":
        F[pick] *= -0.5
    else:
        F[pick, 3] = np.inf
    outs, deferred = [], []
    for dense in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7) for _ in range(members)], lattice=lattice, precision="fp32dev",
                         dx=1.0, r_res=r_res, cell=1.0, moment_capacity=2 * len(X))
        sim.set_dense_stencil(dense)
        sim.set_state(inst, X, F)
        sim.step(1)
        deferred.append(sim.trace("deferred").cpu().numpy().view(np.uint32).tolist())
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    whole = {2: 2 * 5, 3: 8}[len(dims)]  # tiles of 32 x 8 cells, or bricks of 8^3, of one instance
    assert deferred[0] == [0, 0, whole]
