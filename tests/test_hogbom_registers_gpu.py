"""The register-resident FP32 CLEAN loop against the oracle, bit for bit, at the
edges of its variants: one to four column groups, rows per thread from one to
the most, fewer rows than SMs, PSF rows that allow bulk copies and rows that do
not, PSFs larger than the image, a clean box, a mask, peaks at the image's
corners, ties, residuals that are all zero or masked, and the image sizes that
fall back to the shared-memory loop."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(ny, nx, pny, pnx, seed):
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:pny, 0:pnx]
    r2 = (yy - pny // 2) ** 2 + (xx - pnx // 2) ** 2
    psf = (np.exp(-r2 / 8.0) + 0.03 * np.cos(0.7 * np.sqrt(r2))).astype(np.float32)
    dirty = (0.01 * rng.normal(size=(ny, nx))).astype(np.float32)
    for y, x in ((0, 0), (ny - 1, nx - 1), (ny // 2, 0), (0, nx - 1), (ny // 3, nx // 2)):
        dirty[y, x] = 1.0  # ties
    return dirty, psf


SIZES = [(1, 1), (2, 31), (7, 33), (150, 64), (149, 100), (300, 512), (297, 513), (520, 600),
         (149, 1024), (1200, 700), (64, 1025), (300, 1501), (160, 2047), (2072, 2048), (40, 2052)]


@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("large", [False, True])
def test_matches_oracle(ny, nx, large):
    import oracle as O
    from astroviper_b200.core.imaging.deconvolvers import hogbom
    pny, pnx = (ny + 9, nx + 6 + (-nx - 6) % 4) if large else (ny, nx)
    dirty, psf = _case(ny, nx, pny, pnx, ny * 7 + nx)
    rng = np.random.default_rng(1)
    mask = (rng.uniform(size=dirty.shape) < 0.7).astype(np.float32)
    box = (min(1, nx - 1), nx, 0, max(1, ny - 1))
    for kw in (dict(), dict(mask=mask), dict(clean_box=box, speedup=20.0, threshold=1e-3)):
        it = 40
        a = hogbom.clean(dirty, psf, max_iter=it, gain=0.2, large_psf=large, **kw)
        b = O.hogbom_clean(dirty, psf, max_iter=it, gain=0.2, **kw)
        assert a["iterations_performed"] == b["iterations_performed"]
        for k in ("model_image", "residual_image"):
            assert np.array_equal(a[k], b[k]), k


def test_nothing_above_zero():
    import oracle as O
    from astroviper_b200.core.imaging.deconvolvers import hogbom
    d, p = _case(70, 64, 70, 64, 3)
    for dirty, kw in ((np.zeros_like(d), {}), (d, dict(mask=np.zeros_like(d) + 0.25))):
        a = hogbom.clean(dirty, p, max_iter=5, **kw)
        b = O.hogbom_clean(dirty, p, max_iter=5, **kw)
        assert a["iterations_performed"] == b["iterations_performed"]
        assert np.array_equal(a["model_image"], b["model_image"])
        assert np.array_equal(a["residual_image"], b["residual_image"])


@pytest.mark.parametrize("n", [1, 1000, 16384, 16385, 100_000, 20_000_000])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_extremes_and_ordered_sum(n, dt):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(n)
    x = rng.normal(size=(1, n)).astype(dt)
    x[0, rng.uniform(size=n) < 0.9] = 0.0
    s = dt(0)
    for v in np.abs(x[x != 0])[:200_000]:
        s = dt(s + v)
    if n <= 1_000_000:
        assert K.abs_sum_ordered(x).cpu().numpy()[0] == s
    for y in (x, np.abs(x) + dt(1), -np.abs(x) - dt(1)):
        got = K.maximg(y).cpu().numpy()
        assert got[0] == y.min() and got[1] == y.max()
    m = (rng.uniform(size=x.shape) < 0.5).astype(dt)
    if m.any():
        got = K.maximg(x, m).cpu().numpy()
        assert got[0] == x[m > 0.5].min() and got[1] == x[m > 0.5].max()
    x[0, 0] = np.nan
    got = K.maximg(x).cpu().numpy()
    if n > 1:
        assert got[0] == np.nanmin(x) and got[1] == np.nanmax(x)
