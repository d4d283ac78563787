"""Stage functions where a coordinate is so many cells off that its quotient by dx overflows: points at one
place are still within dx of each other."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x0", [1.0e30, -1.0e30, 1.0e25, 3.0])
def test_resample_at_overflowing_quotients(x0):
    from direbm_gb300 import warp as w
    from oracle.lattices import D2Q7

    dx = 1.0e-9
    cp = np.array([[x0, 0.5], [x0, -2.0], [0.25, x0]], dtype=np.float32)
    rng = np.random.default_rng(2)
    val = rng.uniform(0.1, 1.0, (3, D2Q7.Q)).astype(np.float32)
    pos_c = np.repeat(cp, D2Q7.Q, axis=0)
    dirs = np.tile(np.arange(D2Q7.Q, dtype=np.int32), 3)
    pos, out = w.resample(pos_c, val.reshape(-1), dirs, cp, dx, np.asarray(D2Q7.W, np.float32))
    np.testing.assert_array_equal(pos.numpy(), cp)
    # one control point per place: every component's whole value goes to it, (dx - 0) / dx = 1
    np.testing.assert_array_equal(out.numpy(), val)
    # the refine sees all seven directions there and moves to their centroid: the place itself, to the rounding
    # of a weighted mean
    new = w.refine_control_points(cp, pos_c, val.reshape(-1), dirs, dx, 4).numpy()
    np.testing.assert_allclose(new, cp, rtol=1e-6)
