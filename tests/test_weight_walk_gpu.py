"""The weight kernels' walk (a thread per (baseline, channel) series and block
of times) against a plain restatement, at its edges: one time step and one
series, odd numbers of times, more channels than a
block's 256 threads, more series than one block, all polarisation counts and
types, flags, NaN weights and samples off the grid.  Weights are multiples of
1/64, so every sum is exact in FP64 and the grids must be equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

C_LIGHT = 299792458.0
CELL = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8


def _restate(uvw, freq, w, n, cell):
    nchan = len(freq)
    g = np.zeros((nchan, 1) + n)
    sw = np.zeros((nchan, 1))
    places = np.full(w.shape[:3] + (2,), -1)
    for t, b, c in np.ndindex(*w.shape[:3]):
        pos = [uvw[t, b, k] * (-(freq[c] * cell[k] * n[k]) / C_LIGHT) for k in (0, 1)]
        if np.isnan(pos).any():
            continue
        at = [int(pos[k] + n[k] // 2 + 0.5) for k in (0, 1)]
        cj = [int(-pos[k] + n[k] // 2 + 0.5) for k in (0, 1)]
        if not all(0 <= at[k] < n[k] for k in (0, 1)):
            continue
        places[t, b, c] = at
        if np.isnan(w[t, b, c]):
            continue
        g[c, 0, at[0], at[1]] += w[t, b, c]
        if all(0 <= cj[k] < n[k] for k in (0, 1)):
            g[c, 0, cj[0], cj[1]] += w[t, b, c]
        sw[c, 0] += 2.0 * w[t, b, c]
    return g, sw, places


@pytest.mark.parametrize("nt,nb,nchan", [(1, 1, 1), (5, 1, 3), (7, 3, 300), (64, 90, 3),
                                         (4, 257, 1)])
@pytest.mark.parametrize("npol", [1, 2, 4])
@pytest.mark.parametrize("wdt,odt", [(np.float32, torch.float64), (np.float64, torch.float32)])
def test_density_and_briggs_weights(nt, nb, nchan, npol, wdt, odt):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(nt * 1000 + nb + nchan + npol)
    n = (41, 64)
    uvw = np.cumsum(rng.normal(size=(nt, nb, 3)) * 60.0, axis=0) + rng.normal(size=(nb, 3)) * 400
    if nt > 1:
        uvw[1, 0, 0] = np.nan
    freq = np.linspace(1.0e9, 1.4e9, nchan)
    wt = (rng.integers(0, 128, (nt, nb, nchan, npol)) / 64.0).astype(wdt)
    if nt > 2:
        wt[2, 0, 0, 0] = np.nan
    flag = rng.uniform(size=wt.shape) < 0.1
    w = np.where(flag, np.nan, wt.astype(np.float64))
    w = {1: w[..., 0], 2: (w[..., 0] + w[..., npol - 1]) / 2,
         4: (w[..., 0] + w[..., npol - 1]) / 2}[npol]
    g, sw, places = _restate(uvw, freq, w, n, CELL)
    gd, sd = K.weight_density(uvw, freq, wt, flag, n, CELL)
    assert np.array_equal(gd.cpu().numpy(), g)
    assert np.array_equal(sd.cpu().numpy(), sw)
    fac = np.array([rng.uniform(0.5, 2.0, (nchan, 1)), np.ones((nchan, 1))])
    iw, err = K.briggs_apply(gd, fac, uvw, freq, wt, flag, n, CELL, out_dtype=odt)
    ref = np.zeros(w.shape)
    for i in np.ndindex(*w.shape):
        a, b = places[i]
        if a < 0:
            continue
        ref[i] = w[i]
        if not np.isnan(w[i]) and w[i] != 0 and g[i[2], 0, a, b] != 0:
            ref[i] = w[i] / (fac[0, i[2], 0] * g[i[2], 0, a, b] + fac[1, i[2], 0])
    ref = ref.astype(np.float32 if odt == torch.float32 else np.float64)
    assert int(err.item()) == 0
    assert np.array_equal(iw.cpu().numpy(), np.repeat(ref[..., None], npol, -1), equal_nan=True)
    fac[0, 0, 0] = np.nan
    _, err = K.briggs_apply(gd, fac, uvw, freq, wt, flag, n, CELL)
    c0 = places[:, :, 0, 0] >= 0
    hit = c0 & ~np.isnan(w[:, :, 0]) & (w[:, :, 0] != 0)
    assert int(err.item()) == int(any(g[0, 0, a, b] != 0 for a, b in places[:, :, 0][hit]))
