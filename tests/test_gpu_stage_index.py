"""The stage functions' sorted-cell index: table of cell starts, searched keys and full-length keys (captured
streams) give the same bits, and they match the oracle (oracle/stages.py) to the tolerances of its other
stage tests, or four units in the last place of the coordinates where that is more: two rounded sums and a
quotient make about 1.5."""

import numpy as np
import pytest

from oracle import stages
from oracle.physics import equilibrium

pytestmark = pytest.mark.gpu

DX = 0.75


def _points(case, rng):
    x = rng.uniform(-6.0, 6.0, size=(257, 2))
    if case == "cell_borders":  # multiples of the cell: columns two away come into reach by rounding
        x = DX * rng.integers(-5, 6, size=(257, 2)).astype(np.float64)
    if case == "crowded":
        x[:150] = x[0] + rng.uniform(-0.05, 0.05, size=(150, 2))
    if case == "line":
        x[:, 0] = 0.25
    if case == "single":
        x = x[:1]
    if case == "far":  # thousands of cells off: the quotients' rounding grows
        x = x + [40000.0, -70000.0]
    return x


@pytest.mark.parametrize("case", ["box", "cell_borders", "crowded", "line", "single", "far"])
def test_stage_index(case):
    import torch

    from direbm_gb300 import warp as w

    rng = np.random.default_rng(7)
    x = _points(case, rng)
    u = 0.05 * np.sin(x)
    f = equilibrium(rng.uniform(0.3, 1.2, size=len(x)), u).astype(np.float32)
    f_rest = equilibrium(np.float64(1.0), np.zeros(2))
    atol = max(2e-5, 4 * float(np.spacing(np.float32(np.abs(x).max()))))

    def run(x, f):
        pc, vc, dc = w.disperse(x, f, dx=DX)
        cp, p = w.create_control_points(pc, 0.25)
        new = w.refine_control_points(cp, pc, vc, dc, DX, 4)
        pos, out = w.resample(pc, vc, dc, new, DX, f_rest)
        return (pc, vc, dc), [t.numpy() for t in (cp, new, pos, out)]

    comps, (cp, new, pos, out) = run(x, f)
    pc, vc, dc = (c.numpy() for c in comps)
    cp_o, _, _, _ = stages.create_control_points(pc, 0.25)
    np.testing.assert_array_equal(cp, cp_o)
    new_o, _ = stages.refine_control_points(cp, pc, vc, dc, DX, 4)
    np.testing.assert_allclose(new, new_o, rtol=0, atol=atol)
    _, f_o, _ = stages.resample(pc, vc, dc, new, DX, f_rest)
    np.testing.assert_array_equal(pos, new)
    np.testing.assert_allclose(out, f_o, rtol=2e-5, atol=1e-6)

    # a moment far away leaves the table of starts for searched keys: the other points' bits stay
    far = np.concatenate([x, [[3.0e6, 2.0e6]]])
    _, (cp2, new2, pos2, out2) = run(far, np.concatenate([f, f[:1]]))
    here = np.abs(cp2[:, 0]) < 1e6
    for a, b in ((cp, cp2), (new, new2), (pos, pos2), (out, out2)):
        np.testing.assert_array_equal(a, b[here])

    # a captured stream allows no look at the bounds: keys of full length
    s = torch.cuda.Stream()
    w.refine_control_points(cp, *comps, DX, 4)
    cp_t = torch.as_tensor(cp, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        r = w.refine_control_points(cp_t, *comps, DX, 4)
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(r.numpy(), new)
