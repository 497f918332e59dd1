"""Samples that the mosaic gridder skips (zero or NaN weight, NaN data, no
function, no image polarisation) touch no cell, whatever the convolution
functions hold: with NaN and infinite taps in the first function (which no
sample may use) and in a used one, the register kernel gives the finite cells
of the per-sample kernel.  Both add FP64 products of a few hundred samples in
another order: 1e-13 of the largest cell."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_support", [3, 6, 9, 11])
@pytest.mark.parametrize("npol,n_cfp", [(1, 1), (2, 1), (2, 2), (3, 3), (4, 1), (4, 2)])
@pytest.mark.parametrize("do_psf", [False, True])
@pytest.mark.parametrize("spread", [0, 2])
def test_skipped_samples_read_no_taps(max_support, npol, n_cfp, do_psf, spread):
    """spread: the used function's bad taps are those of one kernel offset, or
    of every offset (2 = os // 2)."""
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(max_support * 100 + npol * 10 + n_cfp)
    nt, nb, nchan, os_, n_cfb, n_cfc = 9, 6, 3, 4, 4, 2
    n = (max_support + 1) * os_
    cf = rng.normal(size=(n_cfb, n_cfc, n_cfp, n, n)) + 1j * rng.normal(
        size=(n_cfb, n_cfc, n_cfp, n, n))
    cf[0] = np.nan
    mid = slice(n // 2 - spread, n // 2 + spread + 1)
    cf[1, 0, 0, mid, mid] = np.inf
    cf[1, 1, -1, mid, n // 2 + os_ - spread:n // 2 + os_ + spread + 1] = complex(1.0, np.nan)
    sup = np.full((n_cfb, n_cfc, n_cfp, 2), max_support)
    sup[2, :, :, 0] = max(1, max_support - 2)
    uvw = rng.normal(size=(nt, nb, 3)) * 500.0
    shape = (nt, nb, nchan, npol)
    vis = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    wt = rng.uniform(0.5, 2.0, size=shape)
    wt[rng.uniform(size=shape) < 0.2] = 0.0
    wt[rng.uniform(size=shape) < 0.1] = np.nan
    vis[rng.uniform(size=shape) < 0.1] = np.nan
    wt[4] = 0.0
    vis[5, :, 1] = np.nan
    freq = np.array([1.0e9, 1.1e9, 1.3e9])
    cell = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8
    # baselines on the poisoned functions, on sound ones and on none
    cfb, cfc = np.array([2, 3, 1, -1, 2, 3]), np.array([0, 1, 1])
    pm, cfp = np.arange(npol)[::-1].copy(), np.arange(npol) % n_cfp
    if npol == 3:
        pm[1] = -1
    out = []
    for tiled in (False, True):
        grid = torch.zeros((2, npol, 201, 178), dtype=torch.complex128, device="cuda")
        sw = torch.zeros((2, npol), dtype=torch.float64, device="cuda")
        K.mosaic_grid(grid, sw, do_psf, vis, wt, uvw, freq, np.array([0, 1, 0]), pm, cfb, cfc,
                      cfp, torch.as_tensor(cf, device="cuda"), sup, (201, 178), cell, os_,
                      tiled=tiled)
        out.append((torch.view_as_real(grid).cpu().numpy(), sw.cpu().numpy()))
    (ga, sa), (gb, sb) = out
    for x, y in ((ga, gb), (sa, sb)):
        ok = np.isfinite(x)
        assert np.array_equal(ok, np.isfinite(y))
        assert np.abs(y[ok] - x[ok]).max(initial=0.0) <= 1e-13 * np.abs(x[ok]).max(initial=0.0) + (
            1e-12 * np.nansum(wt) if x is sa else 0.0)
    assert np.abs(ga[np.isfinite(ga)]).max() > 0
    assert spread == 0 or not np.isfinite(ga).all()
