"""The sort-free placement of control points in a simulator that held another, denser state before."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32dev", "fp64"])
@pytest.mark.parametrize("lattice", ["D2Q9", "D2Q7"])
@pytest.mark.parametrize("dense", [True, False])
def test_sparse_state_after_dense_state(lattice, precision, dense):
    """A cell without a control point keeps no refined cell of an earlier step: a sparse state stepped in
    a used simulator gives the bits of the same state in a new one, with no status bit."""
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    lat = get(lattice)
    n = 40
    rng = np.random.default_rng(3)
    c = np.stack(np.meshgrid(np.arange(n), np.arange(n)), -1).reshape(-1, 2).astype(np.float64)
    full = c + rng.uniform(0.2, 0.8, c.shape)
    sparse = c[::17] + rng.uniform(0.05, 0.95, c[::17].shape)

    def f_of(x):
        return equilibrium(np.ones(len(x)), 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 0])], 1), lat)

    outs = []
    for used in (False, True):
        sim = Simulation([Instance(dims=(n, n), tau=0.7)], lattice=lattice, precision=precision, dx=1.0, r_res=1.5,
                         cell=1.0)
        sim.set_dense_stencil(dense)
        if used:
            sim.set_state(None, full, f_of(full))
            sim.step(3)
        sim.set_state(None, sparse, f_of(sparse))
        sim.step(3)
        assert sim.status() == 0
        outs.append(sim.state_numpy())
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
