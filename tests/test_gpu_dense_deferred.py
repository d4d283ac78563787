"""Dense tiles handed to the row segments: their control points are emitted after the gather, by the pass that
takes the points with gaps.  Bits against the row segments alone."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sim(lattice, dx, r_res, x, f, dims, dense, precision="fp32dev"):
    from direbm_gb300.sim import Instance, Simulation

    sim = Simulation([Instance(dims=dims, tau=0.7)], lattice=lattice, precision=precision, dx=dx, r_res=r_res, cell=1.0,
                     moment_capacity=2 * len(x) + dims[0] * dims[1])
    sim.set_dense_stencil(dense)
    sim.set_state(None, x, f)
    return sim


def _state(lattice, dims, crowd, seed=5):
    from direbm_gb300.lattices import get
    from oracle.physics import equilibrium

    rng = np.random.default_rng(seed)
    c = np.stack(np.meshgrid(np.arange(dims[0]), np.arange(dims[1]), indexing="ij"), -1).reshape(-1, 2).astype(float)
    more = c[rng.integers(0, len(c), int(crowd * len(c)))]
    few = c[c[:, 0] < dims[0] // 3]  # a crowded third beside regular tiles
    c = np.concatenate([c, few[rng.integers(0, len(few), len(few) // 2)], more])
    x = c + rng.uniform(0.02, 0.98, c.shape)
    u = 0.03 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 0])], 1)
    return x, equilibrium(np.ones(len(x)), u, get(lattice))


@pytest.mark.parametrize("lattice,dx,r_res", [("D2Q9", 1.0, 1.5), ("D2Q9", 1.0, 1.9), ("D2Q9", 1.0, 0.9),
                                              ("D2Q9", 2.0, 1.5), ("D2Q7", 1.0, 1.5), ("D2Q7", 4.0, 4.0)])
@pytest.mark.parametrize("dims", [(40, 37), (200, 150)])  # directions of a tile shared by blocks, and not
def test_deferred_tiles(lattice, dx, r_res, dims):
    x, f = _state(lattice, dims, 0.02)
    outs = []
    for dense in (True, False):
        sim = _sim(lattice, dx, r_res, x, f, dims, dense)
        sim.step(3)
        p = sim.count()
        empty = sim.trace("empty").cpu().numpy().view(np.uint32)[:p]
        assert (empty < 1 << 9).all()  # directions alone
        outs.append(sim.state_numpy() + (empty, np.int64(sim.status())))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
