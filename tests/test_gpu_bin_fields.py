"""Binned mass and momentum, bit for bit: a moment's sums term by term from k = 0, a bin's sums in input
order, every operation rounded to FP64, bins by numpy's rule (searchsorted)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(kind, rng):
    e = np.arange(-3.0, 4.0 + 0.7, 0.7)
    if kind == "uneven":
        e = np.sort(np.concatenate([rng.uniform(-3, 4, 9), [-3.0, 4.0, 0.0]]))
    if kind == "repeated":
        e = np.sort(np.concatenate([e, e[3:5]]))
    if kind == "two":
        e = e[[0, -1]]
    if kind == "far":  # the proportion in FP32 is off by many bins
        e = 1.0e9 + e
    return e


@pytest.mark.parametrize("lattice", ["D2Q9", "D2Q7", "D3Q19", "D3Q13"])
@pytest.mark.parametrize("kind", ["even", "uneven", "repeated", "two", "far", "not_finite"])
def test_bin_fields_bits(kind, lattice):
    from direbm_gb300.fields import bin_fields3_device, bin_fields_device
    from direbm_gb300.lattices import get

    lat = get(lattice)
    D, Q = lat.D, lat.Q
    c = np.asarray(lat.C, np.float64)
    rng = np.random.default_rng(13)
    edges = [_edges(kind, rng) for _ in range(D)]
    n = 1031
    x = rng.uniform(-3.3, 4.9, (n, D)) + (1.0e9 if kind == "far" else 0.0)
    for a in range(D):  # on the edges, on the last one, beyond
        x[:40, a] = rng.choice(edges[a], 40)
    x[40] = [e[-1] for e in edges]
    x[41] = -0.0
    x[42] = np.nan
    x[43] = np.inf
    f = rng.normal(0.3, 0.4, (n, Q))
    if kind == "not_finite":
        f[50, 1], f[60, Q - 1], f[70, 0], f[80, 2] = np.inf, np.nan, -np.inf, 1e308
        f[80, 3] = 1e308

    with np.errstate(all="ignore"):
        mm = np.zeros((n, 1 + D))
        for k in range(Q):
            mm[:, 0] += f[:, k]
            for a in range(D):
                mm[:, 1 + a] += f[:, k] * c[k, a]
        ref = np.zeros((1 + D,) + tuple(len(e) - 1 for e in reversed(edges)))
        for i in range(n):
            b = []
            for a in reversed(range(D)):
                e = edges[a]
                ok = e[0] <= x[i, a] <= e[-1]
                b.append(len(e) - 2 if x[i, a] == e[-1] else int(np.searchsorted(e, x[i, a], "right")) - 1 if ok else None)
            if None not in b:
                for v in range(1 + D):
                    ref[(v, *b)] += mm[i, v]
    run = bin_fields_device if D == 2 else bin_fields3_device
    out = run(x, f, *edges, lattice)
    for v in range(1 + D):
        np.testing.assert_array_equal(out[v].cpu().numpy(), ref[v])


def test_capture_is_refused():
    import torch
    from direbm_gb300.fields import bin_fields_device
    from direbm_gb300.lattices import get

    lat = get("D2Q9")
    x = torch.zeros((4, 2), dtype=torch.float64, device="cuda")
    f = torch.ones((4, lat.Q), dtype=torch.float64, device="cuda")
    edges = np.array([-1.0, 0.5, 1.0])
    mass, _, _ = bin_fields_device(x, f, edges, edges, lat)
    with pytest.raises(RuntimeError, match="captured"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            bin_fields_device(x, f, edges, edges, lat)
    again, _, _ = bin_fields_device(x, f, edges, edges, lat)
    assert torch.equal(mass, again) and float(mass[0, 0]) == 4.0 * lat.Q
