"""Tall narrow images on both sides of the line between the register-resident
CLEAN loop and the shared-memory one (rows of a thread, rows of a band, widths
that are powers of two or not): the loop that runs, and the oracle's result bit
for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,band,registers", [
    (16, 80, True), (16, 81, False), (32, 80, True), (32, 81, False), (64, 112, True),
    (64, 113, False), (128, 56, True), (128, 57, False), (256, 28, True), (256, 29, False),
    (512, 14, True), (512, 15, False), (512, 19, False), (512, 20, True), (100, 113, True),
    (300, 29, True), (2, 300, True)])
def test_route_and_result(nx, band, registers):
    import oracle as O
    from torch.profiler import ProfilerActivity, profile

    from astroviper_b200._lib import lib
    from astroviper_b200.core.imaging.deconvolvers import hogbom
    ny = lib().av_device_sm_count() * band
    rng = np.random.default_rng(nx + band)
    yy, xx = np.mgrid[0:ny, 0:nx]
    r2 = (yy - ny // 2) ** 2 + (xx - nx // 2) ** 2
    psf = (np.exp(-r2 / 8.0) + 0.03 * np.cos(0.7 * np.sqrt(r2))).astype(np.float32)
    dirty = (0.01 * rng.normal(size=(ny, nx))).astype(np.float32)
    dirty[[0, ny // 3, ny - 1], [0, nx // 2, nx - 1]] = 1.0
    hogbom.clean(dirty, psf, max_iter=1)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        a = hogbom.clean(dirty, psf, max_iter=12, gain=0.2)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "k_hogbom" in e.name]
    assert names and all(("k_hogbom_reg" in n) == registers for n in names)
    b = O.hogbom_clean(dirty, psf, max_iter=12, gain=0.2)
    assert a["iterations_performed"] == b["iterations_performed"]
    for k in ("model_image", "residual_image"):
        assert np.array_equal(a[k], b[k]), k
