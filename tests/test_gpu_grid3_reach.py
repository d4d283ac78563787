"""Displacements longer than the radius in 3D, where a window's exact range holds three cells and the grid
kernels would read a fourth: every bit has to agree with the untiled kernels, and the case has to run on the
kernels whose staged region holds all it reads."""

import numpy as np
import pytest


def _windows_inside(dx, r, c, halo=3, brick=8, tiny=1e-4):
    """Whether the four cells from every window's first one lie in a brick's staged region, per axis, over
    offsets of a point in [0, 1) and the brick's first and last cells (FP32, as the kernels form them)."""
    f = np.float32
    p = np.concatenate([np.linspace(0, 1, 4001), np.nextafter(1.0, 0) * np.ones(1)]).astype(f)
    ok = True
    for cd in {f(v * dx) for v in c}:
        lo = np.floor((p - cd) - f(r) - f(tiny))
        ok &= bool((lo >= -halo).all() and (lo + 3 <= halo).all())
    return ok


def test_the_rule_by_arithmetic():
    """The host's rule (sim.cu, init_brick3), restated, against the windows' cells."""
    for dx in np.arange(0.2, 2.01, 0.05):
        for r in (1.01, 1.05, 1.1, 1.2, 1.3, 1.4, 1.5):
            cd = dx * (1 + 1e-6)
            taken = not (np.floor(-cd - r - 2e-4) < -3 or np.floor(1 + cd + r + 2e-4) > 3
                         or np.floor(1 + cd - r - 5e-5) + 3 > 3)
            if taken:
                assert _windows_inside(dx, r, (-1, 0, 1)), (dx, r)
    assert not _windows_inside(1.5, 1.2, (-1, 0, 1))  # what the exact range alone would accept


@pytest.mark.gpu
@pytest.mark.parametrize("lattice", ["D3Q19", "D3Q13"])
@pytest.mark.parametrize("dx,r_res", [(1.5, 1.2), (1.7, 1.2), (1.25, 1.05), (1.2, 1.2), (1.1, 1.2), (0.5, 1.4)])
def test_long_displacements_equal_untiled(lattice, dx, r_res):
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    dims = (21, 18, 26)
    rng = np.random.default_rng(11)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, 3).astype(np.float64)
    off = rng.uniform(0.0, 1.0, c.shape)
    off[::5] = rng.choice([0.0, 0.9, 0.99, float(np.float32(1) - np.float32(2.0 ** -24))], off[::5].shape)
    x = c + off
    u = 0.02 * np.stack([np.sin(x[:, 1]), np.cos(x[:, 2]), np.sin(x[:, 0])], 1)
    f = equilibrium(np.ones(len(x)), u, get(lattice))
    outs = []
    for grid in (True, False):
        sim = Simulation([Instance(dims=dims, tau=0.7)], lattice=lattice, precision="fp32dev", dx=dx, r_res=r_res,
                         cell=1.0, moment_capacity=2 * len(x))
        sim.set_dense_stencil(grid)
        sim.set_state(None, x, f)
        sim.step(3)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
