"""The dense-stencil kernels of one-cell displacements against the row-segment kernels, at the edges
of what they accept.  Both visit the same hits in the same order, so every bit has to agree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(n0, n1, seed):
    from oracle.lattices import D2Q9
    from oracle.physics import equilibrium

    rng = np.random.default_rng(seed)
    x = np.stack(np.meshgrid(np.arange(n0) + 0.5, np.arange(n1) + 0.5), -1).reshape(-1, 2)
    x = np.mod(x + rng.uniform(-0.45, 0.45, x.shape), [n0, n1])
    u = 0.03 * np.stack([np.sin(2 * np.pi * x[:, 1] / n1), np.cos(2 * np.pi * x[:, 0] / n0)], 1)
    return x, equilibrium(np.ones(len(x)), u, D2Q9), rng


@pytest.mark.parametrize("r_res", [0.9, 1.0, 1.02, 1.3, 1.5, 1.6, 1.95])
@pytest.mark.parametrize("width", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("case", ["jittered", "upper_edge", "around_half", "pairs", "negative_rho", "infinite_f"])
def test_near_dense_equals_row_segments(case, width, r_res):
    """upper_edge: offsets of 1 - 2^-24, which adding one cell carries into the next; around_half:
    offsets within 1e-4 of 1/2 (windows five cells wide at r = 1.5) beside cells with offsets at 0;
    pairs: second moments in 3 % of the cells and none in as many; negative_rho, infinite_f: a moment
    that the gather's sums of non-negative finite terms do not serve."""
    from direbm_gb300.sim import Instance, Simulation

    n0, n1 = 37, 29  # ragged against every tile shape
    x, f, rng = _box(n0, n1, 7)
    c = np.floor(x)
    pick = rng.choice(len(x), len(x) // 8, replace=False)
    if case == "upper_edge":
        x[pick] = c[pick] + np.float64(np.float32(1) - np.float32(2.0 ** -24))
    elif case == "around_half":
        x[pick] = c[pick] + 0.5 + rng.uniform(-1e-4, 1e-4, (len(pick), 2))
        low = rng.choice(len(x), len(x) // 8, replace=False)
        x[low] = c[low] + rng.uniform(0, 1e-4, (len(low), 2))
    elif case == "pairs":
        pick = pick[: len(x) // 32]
        x[pick] = np.mod(c[pick] + [1, 0], [n0, n1]) + rng.uniform(0.1, 0.9, (len(pick), 2))
    elif case == "negative_rho":
        f[pick[0]] *= -0.5
    elif case == "infinite_f":
        f[pick[0], 3] = np.inf
    steps = 1 if case == "infinite_f" else 3
    outs = []
    for dense in (True, False):
        sim = Simulation([Instance(dims=(n0, n1), tau=0.7)], lattice="D2Q9", precision="fp32dev", dx=1.0, r_res=r_res,
                         cell=1.0)
        sim.set_tiling(width, False)
        sim.set_dense_stencil(dense)
        sim.set_state(None, x, f)
        sim.step(steps)
        outs.append(sim.state_numpy() + (np.int64(sim.status()),))
        sim.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
