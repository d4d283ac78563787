"""The stage functions on a captured stream: what synchronises is refused, and leaves the capture whole."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs():
    from direbm_gb300 import warp as w
    from oracle.physics import equilibrium

    rng = np.random.default_rng(4)
    x = rng.uniform(-4.0, 4.0, (200, 2))
    f = equilibrium(np.ones(200), 0.03 * np.sin(x)).astype(np.float32)
    pc, vc, dc = w.disperse(x, f, 1.0)
    cp, _ = w.create_control_points(pc, 0.25)
    rest = torch.tensor([0.5] + [1 / 12] * 6, dtype=torch.float32, device="cuda")
    return w, pc, vc, dc, cp, rest


def test_resample_under_capture_is_refused():
    from direbm_gb300._lib import DbmError

    w, pc, vc, dc, cp, rest = _inputs()
    ref = w.resample(pc, vc, dc, cp, 1.0, rest)[1].numpy()
    t = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t += 1
        with pytest.raises(DbmError, match="captured"):
            w.resample(pc, vc, dc, cp, 1.0, rest)
        t += 1
    g.replay()
    torch.cuda.synchronize()
    assert t.tolist() == [2.0] * 8
    np.testing.assert_array_equal(w.resample(pc, vc, dc, cp, 1.0, rest)[1].numpy(), ref)


def test_resample_without_components_under_capture():
    w, pc, vc, dc, cp, rest = _inputs()
    none = (torch.empty((0, 2), device="cuda"), torch.empty(0, device="cuda"),
            torch.empty(0, dtype=torch.int32, device="cuda"))
    ref = w.resample(*none, cp, 1.0, rest)[1].numpy()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = w.resample(*none, cp, 1.0, rest)[1]
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.numpy(), ref)
