"""The binned FP64 gridder with kernel tables that hold NaN and infinite taps:
the cells and sums of weights that are finite are the plain kernel's, so a
skipped sample (zero or NaN weight, NaN data) and one polarisation of it touch
no cell.  Both add the same FP64 products of a few hundred samples in another
order: 1e-13 of the largest cell.  The degridder's adjoint gives the same cells
in both lane mappings, within 1e-12."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CELL = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8


@pytest.mark.parametrize("support", [3, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("npol", [1, 2, 4])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("do_psf", [False, True])
def test_grid(monkeypatch, support, npol, bad, do_psf):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(support * 10 + npol)
    nt, nb, nchan, os_ = 41, 7, 3, 100
    uvw = rng.normal(size=(nt, nb, 3)) * 400.0
    shape = (nt, nb, nchan, npol)
    vis = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    wt = rng.uniform(0.2, 2.0, shape)
    wt[rng.uniform(size=shape) < 0.3] = 0.0
    wt[3:9] = 0.0
    vis[rng.uniform(size=shape) < 0.1] = np.nan
    # places 0, 28 (read by offset -128 of a support of 3 cells or more) and
    # the last: some samples' taps, and an empty group slot's
    cgk = K.pswf_table(os_, support).cpu().numpy()
    cgk[[0, 28, -1]] = bad
    args = (vis, torch.as_tensor(wt), uvw, np.array([1.0e9, 1.2e9, 1.3e9]), np.array([0, 1, 0]),
            np.arange(npol)[::-1].copy(), cgk, (361, 344), CELL, support, os_, 2, npol)
    out = []
    for binned in (False, True):
        monkeypatch.setattr(K, "_binning_pays", lambda *x, b=binned: b)
        n0 = K.lib().av_launch_count()
        g, s = K.grid(*args, do_psf=do_psf, precision="fp64")
        assert (K.lib().av_launch_count() - n0 > 3) == binned
        out.append((torch.view_as_real(g).cpu().numpy(), s.cpu().numpy()))
    (ga, sa), (gb, sb) = out
    for x, y in ((ga, gb), (sa, sb)):
        ok = np.isfinite(x)
        assert np.array_equal(ok, np.isfinite(y))
        assert np.abs(y[ok] - x[ok]).max(initial=0.0) <= 1e-13 * np.abs(x[ok]).max(initial=0.0)
    assert np.abs(ga[np.isfinite(ga)]).max() > 0 and not np.isfinite(ga).all()


@pytest.mark.parametrize("support", [5, 6, 7, 8])
@pytest.mark.parametrize("npol", [1, 2, 4])
def test_adjoint(support, npol):
    """The adjoint's tensor lanes against its row lanes."""
    from astroviper_b200 import _lib
    from astroviper_b200.forward_model import ForwardModel
    rng = np.random.default_rng(npol)
    uvw = rng.normal(size=(11, 7, 3)) * 400.0
    n = 256
    v = torch.as_tensor(rng.normal(size=(11, 7, 2, npol)) + 1j * rng.normal(size=(11, 7, 2, npol)),
                        device="cuda").to(torch.complex64)
    F = ForwardModel(uvw, np.array([1.0e9, 1.2e9]), (n, n), CELL, npol=npol, support=support)
    F.cgk = F.cgk.clone()
    F.cgk[28] = float("nan")
    out = []
    old = _lib.lib().av_tune_get(_lib.AV_TUNE_GRID_LANES)
    try:
        for lanes in (_lib.AV_GRID_LANES_ROWS, _lib.AV_GRID_LANES_MMA):
            _lib.lib().av_tune_set(_lib.AV_TUNE_GRID_LANES, lanes)
            out.append(torch.view_as_real(F.degrid_adjoint(v)).cpu().numpy())
    finally:
        _lib.lib().av_tune_set(_lib.AV_TUNE_GRID_LANES, old)
    a, b = out
    ok = np.isfinite(a)
    assert np.array_equal(ok, np.isfinite(b))
    assert np.abs(a[ok]).max() > 0
    assert np.abs(a[ok] - b[ok]).max() <= 1e-12 * np.abs(a[ok]).max()
