"""The tiled kernels against the plain FP64 ones called by name, with nothing
in common but the inputs (precision="fp64" runs the binned kernels on the
plans and lanes that the tiled ones use): a slice of the 33M-sample workload
(2048^2 continuum, 4 polarisations), runs of one cell that span many rounds."""
import numpy as np
import pytest
import torch

import bench

pytestmark = pytest.mark.gpu


def _work(n_time, n_chan):
    from astroviper_b200 import _kernels as K
    from astroviper_b200 import synthetic as S
    W = S.workload_large(n_time=n_time, n_chan=n_chan, device=torch.device("cuda"))
    g = torch.Generator("cuda").manual_seed(5)
    wt = torch.rand(W["vis"].shape, dtype=torch.float32, device="cuda", generator=g) + 0.5
    return W, wt, K.pswf_table(100, 7)


@pytest.fixture(params=["mma", "rows"])
def lanes(request):
    from astroviper_b200 import _lib
    L = _lib.lib()
    old = L.av_tune_get(_lib.AV_TUNE_GRID_LANES)
    L.av_tune_set(_lib.AV_TUNE_GRID_LANES, {"mma": _lib.AV_GRID_LANES_MMA,
                                            "rows": _lib.AV_GRID_LANES_ROWS}[request.param])
    yield
    L.av_tune_set(_lib.AV_TUNE_GRID_LANES, old)


@pytest.mark.parametrize("do_psf", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_grid(lanes, precision, do_psf):
    """FP64 sums of the same FP64 products in another order: 1e-12."""
    from astroviper_b200 import _kernels as K
    W, wt, cgk = _work(8, 16)
    npol = wt.shape[3]
    cm = np.zeros(16, int)
    vis = None if do_psf else W["vis"]
    a, sa = bench.plain_grid(vis, wt, W["uvw"], W["freq"], cm, npol, cgk, W["image_size"],
                             W["pixelincr"], 7, 1, do_psf)
    b, sb = K.grid(vis, wt, W["uvw"], W["freq"], cm, np.arange(npol), cgk, W["image_size"],
                   W["pixelincr"], 7, 100, 1, npol, do_psf=do_psf, precision=precision)
    assert a.abs().max() > 0
    assert torch.linalg.norm(b - a) <= 1e-12 * torch.linalg.norm(a)
    assert ((sb - sa).abs() <= 1e-12 * sa.abs()).all()


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("fp64", 1e-13)])
def test_degrid(precision, tol):
    """FP32 taps and sums within 1e-6, FP64 ones within rounding."""
    from astroviper_b200 import _kernels as K
    W, wt, cgk = _work(4, 16)
    npol = wt.shape[3]
    nx, ny = (int(x) for x in W["image_size"])
    cell, cm = W["pixelincr"], np.zeros(16, int)
    g, _ = bench.plain_grid(W["vis"], wt, W["uvw"], W["freq"], cm, npol, cgk, (nx, ny), cell, 7,
                            1)
    a = bench.plain_degrid(g, W["uvw"], W["freq"], cm, npol, cgk, (nx, ny), cell, 7)
    vals = torch.zeros_like(W["vis"] if precision == "fp32" else a)
    b = K.degrid(g, W["uvw"], W["freq"], (-cell[0] * nx, -cell[1] * ny), (nx / 2, ny / 2), cm,
                 np.arange(npol), cgk, 7, 100, values=vals, precision=precision,
                 accumulate=False).to(torch.complex128)
    assert a.abs().max() > 0
    assert torch.linalg.norm(b - a) <= tol * torch.linalg.norm(a)
