"""The refine's index: the call waits for nothing, and its hits and their order are those of the sorted cells."""

import time

import numpy as np
import pytest
import torch

from oracle import stages

pytestmark = pytest.mark.gpu


def test_refine_returns_while_its_stream_is_busy():
    from direbm_gb300 import warp as w

    rng = np.random.default_rng(1)
    x = torch.as_tensor(rng.uniform(0, 8, (300, 2)), dtype=torch.float32, device="cuda")
    f = torch.full((300, 7), 0.1, device="cuda")
    comps = w.disperse(x, f, 1.0)
    cp, _ = w.create_control_points(comps[0], 0.25)
    ref = w.refine_control_points(cp, *comps, 1.0, 4).numpy()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    torch.cuda._sleep(600_000_000)  # about 0.3 s of a spinning kernel ahead of the call
    out = w.refine_control_points(cp, *comps, 1.0, 4)
    returned = time.perf_counter() - t0
    torch.cuda.synchronize()
    finished = time.perf_counter() - t0
    assert finished > 0.1 and returned < 0.5 * finished, (returned, finished)
    np.testing.assert_array_equal(out.numpy(), ref)


# rows that cross a border of blocks (cells 0xB249 + multiples of 2^16) or wrap around the 32-bit word
@pytest.mark.parametrize("y0", [0.0, 0xB249 * 0.5, (0xB249 - 65536) * 0.5, 2.0 ** 31 * 0.5, 37.25])
@pytest.mark.parametrize("n", [1, 33, 511, 513, 4000])
def test_refine_hits(n, y0):
    from direbm_gb300 import warp as w

    rng = np.random.default_rng(n)
    dx = 0.5
    big = abs(y0) > 1e6  # floats are 64 apart there: points at few distinct places
    x = rng.uniform(-4, 4, (n, 2)) if not big else rng.integers(-3, 4, (n, 2)) * np.array([0.25, 128.0])
    x[:, 1] += y0
    cp = np.concatenate([x[: max(1, n // 3)], x[:1] + [0.25, 0.0]]).astype(np.float32)
    pos = np.repeat(x, 7, axis=0).astype(np.float32)
    pos[:, 0] += np.tile(np.linspace(-0.3, 0.3, 7), n).astype(np.float32)
    val = rng.uniform(0.0, 1.0, 7 * n).astype(np.float32)
    dirs = np.tile(np.arange(7, dtype=np.int32), n)
    new = w.refine_control_points(cp, pos, val, dirs, dx, 3).numpy()
    ref, _ = stages.refine_control_points(cp, pos, val, dirs, dx, 3)
    # two sums, each rounded once, and a quotient: three units in the last place of the coordinate
    atol = 3 * np.spacing(np.maximum(np.abs(cp).max(axis=0), 1.0).astype(np.float32))
    assert (np.abs(new.astype(np.float64) - ref) <= atol).all()
