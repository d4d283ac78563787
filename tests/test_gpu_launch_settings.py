"""Launch settings act where the library says they do: bits per setting on the kernels it reaches, and the
autotuner times that setting."""

import numpy as np
import pytest

from tests._cases import periodic_tg

pytestmark = pytest.mark.gpu


def _sim(lattice, dims, precision, r_res=1.5, **extra):
    from direbm_gb300.sim import Instance, Simulation

    x, f = periodic_tg(dims[0], lattice, seed=6, u0=0.04)
    if "obstacle" in extra:
        center, radius = extra["obstacle"]
        keep = ((x - np.asarray(center)) ** 2).sum(1) > (radius + 0.5) ** 2
        x, f = x[keep], f[keep]
    sim = Simulation([Instance(dims=dims, tau=0.7, **extra)], lattice=lattice, precision=precision, dx=1.0, r_res=r_res,
                     cell=1.0, moment_capacity=2 * len(x))
    sim.set_state(None, x, f)
    return sim


def test_window_path():
    ball2, ball3 = ((20.0, 20.0), 4.0), ((12.0, 12.0, 12.0), 2.0)
    assert _sim("D2Q9", (40, 40), "fp32dev").window_path() == "tiles"
    assert _sim("D2Q7", (40, 40), "fp32dev").window_path() == "tiles"
    assert _sim("D2Q9", (40, 40), "fp64").window_path() == "bricks"
    assert _sim("D2Q9", (40, 40), "fp32dev", obstacle=ball2).window_path() == "bricks"
    assert _sim("D3Q19", (24, 24, 24), "fp64").window_path() == "bricks"
    sim = _sim("D3Q19", (24, 24, 24), "fp32dev")
    assert sim.window_path() == "grid3"
    sim.set_dense_stencil(False)
    assert sim.window_path() == "bricks"
    assert _sim("D3Q19", (24, 24, 24), "fp32dev", r_res=1.8).window_path() == "bricks"
    assert _sim("D3Q19", (24, 24, 24), "fp32dev", obstacle=ball3).window_path() == "bricks"  # all near the sphere


@pytest.mark.parametrize("lattice,dims,precision,widths", [("D3Q19", (24, 24, 24), "fp32dev", (4, 8, 16, 32)),
                                                           ("D2Q9", (40, 40), "fp64", (8, 16, 32, 64)),
                                                           ("D2Q7", (40, 40), "fp64", (8, 16, 32, 64))])
def test_brick_widths_on_the_kernels_they_reach(lattice, dims, precision, widths):
    """3D FP32 by the untiled kernels; 2D FP64 with the placement that needs no sort."""
    sim = _sim(lattice, dims, precision)
    sim.set_dense_stencil(False)
    assert sim.window_path() == "bricks"
    snap = sim.snapshot()
    ref = None
    for w in widths:
        sim.set_brick_width(w)
        sim.restore(snap)
        sim.step(3)
        out = [t.cpu().numpy() for t in sim.state()]
        if ref is None:
            ref = out
        for a, b in zip(out, ref):
            np.testing.assert_array_equal(a, b, err_msg=f"brick {w}")


@pytest.mark.parametrize("lattice,dims,precision,path", [("D2Q9", (40, 40), "fp64", "bricks"),
                                                         ("D3Q19", (24, 24, 24), "fp32dev", "grid3"),
                                                         ("D3Q19", (24, 24, 24), "fp64", "bricks")])
def test_autotuner_times_what_acts(lattice, dims, precision, path, tmp_path, monkeypatch):
    from direbm_gb300 import autotune

    monkeypatch.setenv("DIREBM_GB300_TUNE_CACHE", str(tmp_path / "tiling.json"))
    sim = _sim(lattice, dims, precision)
    before = sim.state_numpy()
    kept = sim.tiling() if len(dims) == 2 else None
    choice = autotune.autotune(sim, steps=1)
    widths = autotune.BRICK_CANDIDATES if len(dims) == 3 else autotune.BRICK_CANDIDATES_2D
    assert choice["path"] == path and not choice["cached"]
    assert set(choice["timings"]) == ({f"brick{w}" for w in widths} if path == "bricks" else {"grid3"})
    assert choice["brick_width"] == sim.brick_width() and choice["brick_width"] in widths
    assert kept is None or sim.tiling() == kept == (choice["tile_width"], choice["persistent"])
    for a, b in zip(before, sim.state_numpy()):
        np.testing.assert_array_equal(a, b)
    sim.set_brick_width(widths[-1])
    again = autotune.autotune(sim, steps=1)
    assert again["cached"] and sim.brick_width() == choice["brick_width"]
