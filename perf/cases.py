"""The work whose speed is followed: passes of the imaging path through its public entry points.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a program
has in hand before the call, run() is one pass, work() its unavoidable bytes and operations and
exact() the same results in 64 bits from plain torch.

A case is a dict of plain values; "kind" says which path it takes:

cycle     a new uv coverage: plan, grid the visibilities, degrid a model (Gridder)
major     one major cycle on a kept plan: residual image, model transform, flagged prediction,
          residual visibilities (Gridder, grid image, FFT helper)
image     grid-corrected images of a stack of gridded planes
double    the FP64 gridder and degridder on complex128 data (precision="fp64")
forward   the differentiable forward model: prediction and its gradient
weights   Briggs weights: density grid, factors, weight of every sample
clean     a Hogbom minor cycle
mosaic    A-projection gridding with per-baseline convolution functions
batched   many independent grids of flagged data in one replayed launch
loop      the whole imaging loop from a measurement set on the host
"""
import math

import numpy as np
import torch

from astroviper_b200 import _kernels as K
from astroviper_b200 import synthetic as S
from astroviper_b200.batched import BatchedGridder
from astroviper_b200.core.imaging.deconvolvers.hogbom import clean
from astroviper_b200.core.imaging.fft import fft_lm_to_uv
from astroviper_b200.core.imaging.imager import run_imaging_loop
from astroviper_b200.core.imaging.imaging_utils.mosaic_grid import mosaic_grid_jit
from astroviper_b200.core.imaging.imaging_utils.standard_degrid import dgrid_numba
from astroviper_b200.core.imaging.imaging_utils.standard_grid import standard_grid_jit
from astroviper_b200.forward_model import ForwardModel
from astroviper_b200.gridder import Gridder

C_LIGHT = 299792458.0
ARCSEC = math.pi / (180.0 * 3600.0)
OVERSAMPLING = 100
MOSAIC_OS, MOSAIC_WINDOW = 4, 12


def listed():
    return [
        # the plain standard gridder at small size: a snapshot of 100,800 samples, where launches
        # and latency count
        dict(name="cycle_small", kind="cycle", ants=64, times=50, chans=1, pols=2, nx=512, ny=512,
             cell=2.0, support=7, cube=False),
        # a small array's spectral cube, one polarisation, sizes that no tile divides
        dict(name="cycle_cube_ragged", kind="cycle", ants=27, times=77, chans=33, pols=1, nx=602,
             ny=754, cell=2.0, support=6, cube=True),
        # the 33M-visibility continuum workload, 4 polarisations, 2048^2
        dict(name="cycle_large", kind="cycle", ants=64, times=256, chans=64, pols=4, nx=2048,
             ny=2048, cell=1.0, support=7, cube=False),
        # one major cycle of an imager that keeps its plan: two polarisations, flagged data
        dict(name="major_flagged", kind="major", ants=64, times=64, chans=16, pols=2, nx=1024,
             ny=1024, cell=1.5, support=7, cube=False),
        # dirty images of four gridded 2048^2 planes
        dict(name="image_4x2048", kind="image", planes=4, nx=2048, ny=2048),
        # complex128 data on the FP64 path, the small array with 8 channels
        dict(name="double_8ch", kind="double", ants=64, times=50, chans=8, pols=2, nx=512, ny=512,
             cell=2.0, support=7),
        # forward and backward pass of the differentiable model, 4.16M visibilities
        dict(name="forward_4M", kind="forward", ants=128, times=128, chans=4, nx=1024, ny=1024,
             cell=1.0, support=7),
        # Briggs weighting of 4.1M samples x 4 polarisations, a density plane per channel
        dict(name="weights_4M", kind="weights", ants=64, times=64, chans=32, pols=4, nx=1024,
             ny=1024, cell=1.5),
        # 1000 minor-cycle iterations on a 2048^2 image
        dict(name="clean_2048", kind="clean", nx=2048, iters=1000),
        # 1.03M samples with convolution functions of two dish sizes
        dict(name="mosaic_1M", kind="mosaic", ants=64, times=64, chans=8, pols=2, nx=1024, ny=1024,
             cell=2.0, small=5, large=7),
        # 128 independent 1024^2 grids of unevenly flagged data, new data each call
        dict(name="batched_128", kind="batched", ants=64, times=248, chans=64, pols=2, nx=1024,
             ny=1024, cell=2.0, support=7),
        # the major / minor-cycle loop on the small measurement set, in double precision
        dict(name="loop_small", kind="loop", times=50, nx=512, ny=512, cell=2.0, niter=1000,
             nmajor=5),
    ]


# the kinds in the proportions in which they are drawn
_DRAWN = ("cycle", "cycle", "cycle", "major", "image", "double", "forward", "weights", "clean",
          "mosaic", "batched", "loop")


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edge(rng, lo, hi):
    """An image edge: a power of two, a multiple of 4 or any number."""
    n = _log(rng, lo, hi)
    how = rng.randrange(3)
    if how == 0:
        return min(hi, max(lo, 1 << round(math.log2(n))))
    return n - n % 4 if how == 1 else n


def _coverage(rng, samples, ants=(16, 128), chans=(1, 64)):
    """Antennas, times and channels of about `samples` samples."""
    a = _log(rng, *ants)
    c = min(_log(rng, *chans), max(1, samples // (a * (a - 1) // 2)))
    t = max(1, min(600, samples // (c * (a * (a - 1) // 2))))
    return dict(ants=a, times=t, chans=c)


def draw(rng):
    kind = rng.choice(_DRAWN)
    if kind == "image":
        return dict(kind=kind, planes=rng.choice((1, 2, 3, 4)), nx=_edge(rng, 256, 2048),
                    ny=_edge(rng, 256, 2048))
    if kind == "clean":
        return dict(kind=kind, nx=_edge(rng, 128, 2048), iters=_log(rng, 100, 1000))
    if kind == "loop":
        n = rng.choice((256, 320, 384, 500, 512))
        return dict(kind=kind, times=_log(rng, 8, 50), nx=n, ny=n, cell=2.0,
                    niter=_log(rng, 100, 1000), nmajor=rng.randint(2, 5))
    n = _edge(rng, 400, 1024 if kind != "cycle" else 2048)
    m = n if rng.random() < 0.5 else _edge(rng, 400, 1024)
    if kind in ("cycle", "major"):
        # even edges: where the gridder's centre n // 2 and the degridder's n / 2 are one, the
        # two directions share a uv coverage
        n, m = n + n % 2, m + m % 2
    # a field that holds the 2 km array's longest baselines at 1.5 GHz with some room
    case = dict(kind=kind, nx=n, ny=m, cell=round(rng.uniform(0.5, 1.0) * 1000.0 / max(n, m), 3))
    if kind == "cycle":
        case.update(_coverage(rng, _log(rng, 20_000, 8_000_000)))
        case.update(pols=rng.choice((1, 2, 4, 4)), support=rng.choice((5, 6, 7, 7, 7, 8)),
                    cube=case["chans"] <= 16 and rng.random() < 0.4)
    elif kind == "major":
        case.update(_coverage(rng, _log(rng, 20_000, 4_000_000)))
        case.update(pols=rng.choice((1, 2, 4)), support=rng.choice((5, 7, 7, 8)), cube=False)
    elif kind == "double":
        case.update(_coverage(rng, _log(rng, 20_000, 800_000), chans=(1, 16)))
        case.update(pols=rng.choice((1, 2, 4)), support=rng.choice((5, 7, 7, 8, 9)))
    elif kind == "forward":
        case.update(_coverage(rng, _log(rng, 50_000, 4_000_000), chans=(1, 8)))
        case.update(support=rng.choice((5, 7, 7, 8)))
    elif kind == "weights":
        case.update(_coverage(rng, _log(rng, 50_000, 4_000_000), chans=(1, 32)))
        case.update(pols=rng.choice((1, 2, 4)))
    elif kind == "mosaic":
        case.update(_coverage(rng, _log(rng, 50_000, 1_000_000), chans=(1, 8)))
        small = rng.choice((3, 5, 7))
        case.update(pols=rng.choice((1, 2)), small=small, large=small + rng.choice((0, 2, 4)))
    else:
        case.update(_coverage(rng, _log(rng, 500_000, 16_000_000), chans=(8, 64)))
        case.update(pols=rng.choice((1, 2)), support=rng.choice((7, 7, 9)))
    return case


# ------------------------------------------------------------------ inputs --
class _Data:
    """Named values."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(1_000_003 + int(seed))
    return g


def _sampling(case, seed, vis_dtype, noise=0.01):
    """uvw, frequencies and the visibilities of five point sources with noise."""
    uvw, rng = S.array_uvw(case["ants"], case["times"], seed=10_000 + int(seed))
    chans = case["chans"]
    freq = np.array([1.4e9]) if chans == 1 else np.linspace(1.0e9, 1.5e9, chans)
    cell = case["cell"] * ARCSEC
    incr = np.array([-cell, cell])
    flux, dx, dy = S.random_sources(rng, 5, 0.1, 1.0, 0.2 * min(case["nx"], case["ny"]))
    l, m = S.source_lm(dx, dy, incr)
    vis = None
    if vis_dtype is not None:
        vis = S.point_source_vis(uvw, freq, case.get("pols", 1), flux, l, m, noise, rng,
                                 dtype=vis_dtype, device=_dev())
    return _Data(uvw=torch.as_tensor(uvw, device=_dev()), freq=freq, incr=incr, vis=vis, rng=rng)


def _sky(case, seed, planes, dtype=torch.float64):
    """Model images: 40 point sources and a few broad blobs in the inner field."""
    g = _gen(seed + 17)
    nx, ny = case["nx"], case["ny"]
    img = torch.zeros((planes, nx, ny), dtype=torch.float64, device=_dev())
    ix = (torch.rand(planes, 40, generator=g, device=_dev()) * 0.7 + 0.15) * nx
    iy = (torch.rand(planes, 40, generator=g, device=_dev()) * 0.7 + 0.15) * ny
    flux = 10.0 ** (torch.rand(planes, 40, generator=g, device=_dev(), dtype=torch.float64) * 2 - 2)
    which = torch.arange(planes, device=_dev())[:, None].expand(-1, 40)
    img.index_put_((which, ix.long(), iy.long()), flux, accumulate=True)
    x = torch.arange(nx, device=_dev(), dtype=torch.float64)[:, None]
    y = torch.arange(ny, device=_dev(), dtype=torch.float64)[None, :]
    for k in range(3):
        cx, cy = ix[:, k, None, None].double(), iy[:, k, None, None].double()
        img += 0.01 * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2.0 * (3.0 + k) ** 2))
    return img.to(dtype)


def _centred_fft(img):
    return torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(img, dim=(-2, -1))),
                              dim=(-2, -1))


def _weight(shape, seed, dtype=torch.float32):
    return torch.rand(shape, generator=_gen(seed + 29), device=_dev(), dtype=dtype) * 0.7 + 0.3


def _planes(case):
    return case["chans"] if case.get("cube") else 1


def _inputs(case, seed):
    """The arrays of a pass, made from the seed alone."""
    kind = case["kind"]
    nx, ny, pols = case["nx"], case.get("ny", case["nx"]), case.get("pols", 1)
    if kind in ("cycle", "major"):
        d = _sampling(case, seed, np.complex64)
        d.weight = _weight(d.vis.shape, seed)
        d.sky = _sky(case, seed, _planes(case) * pols).reshape(_planes(case), pols, nx, ny)
        d.flag = None
        if kind == "major":
            # whole samples and single correlations, 3 % in all
            u = torch.rand(d.vis.shape[:3], generator=_gen(seed + 31), device=_dev())
            v = torch.rand(d.vis.shape, generator=_gen(seed + 37), device=_dev())
            d.flag = (u < 0.02)[..., None] | (v < 0.01)
            d.weight = torch.where(d.flag, torch.zeros_like(d.weight), d.weight)
        return d
    if kind == "image":
        g = _gen(seed)
        shape = (1, case["planes"], nx, ny)
        taper = (torch.hann_window(nx, dtype=torch.float64, device=_dev())[:, None]
                 * torch.hann_window(ny, dtype=torch.float64, device=_dev())[None, :]) ** 4
        grid = torch.randn(shape, generator=g, dtype=torch.complex128, device=_dev()) * taper
        sw = torch.rand((1, case["planes"]), generator=g, dtype=torch.float64, device=_dev()) + 1e4
        return _Data(grid=grid, sum_weight=sw)
    if kind == "double":
        d = _sampling(case, seed, np.complex128)
        d.weight = _weight(d.vis.shape, seed, torch.float64)
        d.model = _centred_fft(_sky(case, seed, pols).reshape(1, pols, nx, ny))
        return d
    if kind == "forward":
        d = _sampling(case, seed, np.complex64)
        d.sky = _sky(case, seed, 1, torch.float32).reshape(1, 1, nx, ny)
        return d
    if kind == "weights":
        d = _sampling(case, seed, None)
        shape = tuple(d.uvw.shape[:2]) + (case["chans"], pols)
        d.weight = _weight(shape, seed)
        d.flag = torch.rand(shape, generator=_gen(seed + 31), device=_dev()) < 0.03
        return d
    if kind == "clean":
        return _clean_inputs(case, seed)
    if kind == "mosaic":
        return _mosaic_inputs(case, seed)
    if kind == "batched":
        d = _sampling(case, seed, np.complex64)
        frac = torch.rand((case["chans"], pols), generator=_gen(seed + 41), device=_dev()) * 0.6
        u = torch.rand(d.vis.shape, generator=_gen(seed + 43), device=_dev())
        d.weight = (u >= frac).to(torch.float32)
        return d
    raise ValueError(kind)


def _clean_inputs(case, seed):
    """A PSF of the small array's sampling and the dirty image of 50 point sources."""
    n = case["nx"]
    uvw, rng = S.array_uvw(64, 50, seed=10_000 + int(seed))
    uv = torch.as_tensor(uvw[:, :, :2].reshape(-1, 2), device=_dev()) * (1.4e9 / C_LIGHT)
    cell = ARCSEC * 2048.0 / n if n < 2048 else ARCSEC
    i = torch.round(uv * cell * n).long()
    i = i[(i.abs() < n // 2).all(dim=1)]
    i = torch.cat([i, -i]) + n // 2
    g = torch.zeros(n * n, dtype=torch.float64, device=_dev())
    g.index_add_(0, i[:, 0] * n + i[:, 1], torch.ones(len(i), dtype=torch.float64, device=_dev()))
    g = g.reshape(n, n)
    psf = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(g))).real
    psf = psf / psf[n // 2, n // 2]
    lo = n // 8
    ys, xs = rng.integers(lo, n - lo, size=(2, 50))
    flux = np.exp(rng.uniform(np.log(0.005), 0.0, size=50))
    dirty = torch.zeros((n, n), dtype=torch.float64, device=_dev())
    for y, x, f in zip(ys.tolist(), xs.tolist(), flux.tolist()):
        dy, dx = y - n // 2, x - n // 2
        ya, yb, xa, xb = max(0, dy), min(n, n + dy), max(0, dx), min(n, n + dx)
        dirty[ya:yb, xa:xb] += f * psf[ya - dy:yb - dy, xa - dx:xb - dx]
    noise = torch.randn((n, n), generator=_gen(seed), dtype=torch.float64, device=_dev())
    return _Data(dirty=(dirty + 1e-4 * noise).float(), psf=psf.float())


def _mosaic_inputs(case, seed):
    """Data in double precision and the convolution functions of two kinds of antenna."""
    d = _sampling(case, seed, np.complex128, noise=0.1)
    d.weight = _weight(d.vis.shape, seed, torch.float64) * 2.0
    ants = case["ants"]
    i, j = np.triu_indices(ants, k=1)
    d.cfb = (i % 2) + (j % 2)  # small-small, mixed, large-large
    d.cfc = (np.arange(case["chans"]) * 2) // max(1, case["chans"])
    n_cfc = int(d.cfc.max()) + 1
    window = max(MOSAIC_WINDOW, case["large"] + 1)
    n = window * MOSAIC_OS
    x = (np.arange(n) - n // 2) / MOSAIC_OS
    support = np.zeros((3, n_cfc, 1, 2), dtype=int)
    cf = np.zeros((3, n_cfc, 1, n, n), dtype=np.complex128)
    mean = (case["small"] + case["large"]) // 4 * 2 + 1
    for b, s in enumerate((case["small"], mean, case["large"])):
        for c in range(n_cfc):
            half = s / 2.0 * (1.0 + 0.05 * c)
            w = np.where(np.abs(x) < half, np.cos(np.clip(x / half, -1, 1) * np.pi / 2) ** 2, 0.0)
            cf[b, c, 0] = np.outer(w, w) * np.exp(0.1j * np.add.outer(x, 0.5 * x))
            support[b, c] = s
    d.cf, d.support = torch.as_tensor(cf, device=_dev()), support
    ramp = np.exp(2j * np.pi * 0.03 * np.add.outer(x, -0.7 * x))
    d.gradient = torch.as_tensor(ramp[None], device=_dev())
    return d


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loop":
        node, params = S.ms4_small(seed=10_000 + int(seed), n_time=case["times"])
        cell = case["cell"] * ARCSEC
        params.update(image_size=(case["nx"], case["ny"]), cell_size=(cell, cell),
                      niter=case["niter"], nmajor=case["nmajor"], cyclefactor=1.5)
        return _Data(case=case, node=node, params=params)
    d = _inputs(case, seed)
    d.case = case
    size = (case["nx"], case.get("ny", case["nx"]))
    pols, support = case.get("pols", 1), case.get("support", 7)
    if kind in ("cycle", "major"):
        d.gridder = Gridder(d.uvw, d.freq, size, d.incr, pols, support=support,
                            oversampling=OVERSAMPLING,
                            chan_mode="cube" if case["cube"] else "continuum")
        if kind == "cycle":
            d.model = _centred_fft(d.sky)
            d.sky = None
        else:
            d.gridder.plan()
    elif kind == "double":
        d.kernel = K.pswf_table(OVERSAMPLING, support)
        d.values = torch.zeros_like(d.vis)
    elif kind == "forward":
        d.model = ForwardModel(d.uvw, d.freq, size, d.incr, npol=1, support=support,
                               oversampling=OVERSAMPLING)
    elif kind == "batched":
        d.gridder = BatchedGridder(d.uvw, d.freq, size, d.incr, pols, support=support,
                                   oversampling=OVERSAMPLING)
    return d


# -------------------------------------------------------------------- pass --
def run(d):
    case = d.case
    kind = case["kind"]
    if kind == "cycle":
        d.gridder.plan()
        grid, sum_weight = d.gridder.grid(d.vis, d.weight)
        return grid, sum_weight, d.gridder.degrid(d.model)
    if kind == "major":
        grid, sum_weight = d.gridder.grid(d.vis, d.weight)
        image = d.gridder.image(grid, sum_weight)
        predicted = d.gridder.degrid(fft_lm_to_uv(d.sky, [2, 3]), flag=d.flag)
        return image, sum_weight, predicted, K.vis_residual(d.vis, predicted)
    if kind == "image":
        return K.grid_to_image(d.grid, d.sum_weight)
    if kind == "double":
        pols, chans, size = case["pols"], case["chans"], np.array([case["nx"], case["ny"]])
        grid = torch.zeros((1, pols, case["nx"], case["ny"]), dtype=torch.complex128,
                           device=d.vis.device)
        sum_weight = torch.zeros((1, pols), dtype=torch.float64, device=d.vis.device)
        standard_grid_jit(grid, sum_weight, False, False, d.vis, d.uvw, d.freq,
                          np.zeros(chans, dtype=int), np.arange(pols), d.weight, d.kernel, size,
                          d.incr, case["support"], OVERSAMPLING, precision="fp64")
        d.values.zero_()
        dgrid_numba(d.uvw, None, d.values, None, -d.incr * size, size / 2, d.model, d.freq,
                    C_LIGHT, case["support"], OVERSAMPLING, d.kernel, np.zeros(chans, dtype=int),
                    np.arange(pols), precision="fp64")
        return grid, sum_weight, d.values
    if kind == "forward":
        x = d.sky.detach().requires_grad_(True)
        predicted = d.model(x)
        (gradient,) = torch.autograd.grad(predicted, x, predicted.detach() - d.vis)
        return predicted.detach(), gradient
    if kind == "weights":
        size = (case["nx"], case["ny"])
        density, sum_weight = K.weight_density(d.uvw, d.freq, d.weight, d.flag, size, d.incr)
        factors = K.briggs_factors(density, sum_weight, 0.5)
        weights, bad = K.briggs_apply(density, factors, d.uvw, d.freq, d.weight, d.flag, size,
                                      d.incr)
        return density, sum_weight, factors, weights, bad
    if kind == "clean":
        r = clean(d.dirty, d.psf, max_iter=case["iters"], gain=0.1, threshold=1e-4)
        return (r["model_image"], r["residual_image"], r["iterations_performed"],
                r["final_peak"], r["total_flux_cleaned"])
    if kind == "mosaic":
        pols, chans = case["pols"], case["chans"]
        grid = torch.zeros((chans, pols, case["nx"], case["ny"]), dtype=torch.complex128,
                           device=d.vis.device)
        sum_weight = torch.zeros((chans, pols), dtype=torch.float64, device=d.vis.device)
        mosaic_grid_jit(grid, sum_weight, False, d.vis, d.uvw, d.freq, np.arange(chans),
                        np.arange(pols), d.cfb, d.cfc, np.zeros(pols, dtype=int), d.weight, d.cf,
                        (case["nx"], case["ny"]), d.incr, d.support,
                        np.array([MOSAIC_OS, MOSAIC_OS]), d.gradient)
        return grid, sum_weight
    if kind == "batched":
        return d.gridder(d.vis, d.weight)
    model, residual, _, _ = run_imaging_loop(d.node, d.params, precision="fp64")
    return model, residual


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes (each input read once, each output written once) and operations of a pass."""
    kind = case["kind"]
    nx, ny = case["nx"], case.get("ny", case["nx"])
    pix = nx * ny
    pols = case.get("pols", 1)
    taps = case.get("support", 7) ** 2
    fft = 5.0 * pix * math.log2(max(2, pix)) / 2  # of real data, or to a real image
    if kind == "image":
        p = case["planes"]
        return {"bytes": p * pix * 24.0, "flops": p * fft}
    if kind == "clean":
        # the residual and PSF pass of an iteration is what CLEAN does; they stay on the chip
        return {"bytes": 4.0 * pix * 4, "flops": 4.0 * pix * case["iters"]}
    if kind == "loop":
        n = 2016.0 * case["times"] * 2
        per = n * (24 + 16 * 4) + 2 * pix * 16 * 4
        return {"bytes": case["nmajor"] * per,
                "flops": case["nmajor"] * (16.0 * taps * n + 4 * fft)}
    tb = case["ants"] * (case["ants"] - 1) / 2.0 * case["times"]
    rows = tb * case["chans"]
    corr = rows * pols
    if kind in ("cycle", "major"):
        cells = float(_planes(case) * pols * pix)
        if kind == "cycle":  # vis, weight, uvw in; grid out; model grid in; values out
            return {"bytes": 20 * corr + 24 * tb + 32 * cells, "flops": 8.0 * taps * corr}
        return {"bytes": 29 * corr + 24 * tb + 16 * cells,
                "flops": 8.0 * taps * corr + 2 * pols * fft}
    if kind == "double":
        return {"bytes": 40 * corr + 24 * tb + 32.0 * pols * pix, "flops": 8.0 * taps * corr}
    if kind == "forward":
        return {"bytes": 16 * corr + 24 * tb + 8.0 * pix, "flops": 8.0 * taps * corr + 2 * fft}
    if kind == "weights":
        used = {1: 1, 2: 2, 4: 2}[pols]
        return {"bytes": rows * (5 * used + 8 * pols) + 24 * tb + 8.0 * case["chans"] * pix,
                "flops": 30.0 * rows}
    if kind == "mosaic":
        s = (case["small"] + case["large"]) / 2
        return {"bytes": 24 * corr + 24 * tb + 16.0 * case["chans"] * pols * pix,
                "flops": 10.0 * s * s * corr}
    return {"bytes": 12 * corr + 24 * tb + 16.0 * case["chans"] * pols * pix,
            "flops": 4.0 * taps * corr * 0.7}


# ------------------------------------------------------- results in 64 bits --
def _spheroidal(u):
    """Schwab's rational approximation of the prolate spheroidal function (m = 6, alpha = 1)."""
    p = np.array([[8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1],
                  [4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2]])
    q = np.array([[1.0, 8.212018e-1, 2.078043e-1], [1.0, 9.599102e-1, 2.918724e-1]])
    u = np.abs(np.asarray(u, dtype=np.float64))
    part = (u >= 0.75).astype(int)
    d = u ** 2 - np.where(part == 1, 1.0, 0.75) ** 2
    top = sum(p[part, k] * d ** k for k in range(5))
    bot = sum(q[part, k] * d ** k for k in range(3))
    return np.where(u <= 1.0, top / bot, 0.0)


def _kernel(support):
    half = support // 2
    u = np.arange(OVERSAMPLING * half) / (half * OVERSAMPLING)
    k = np.concatenate([(1.0 - u ** 2) * _spheroidal(u), np.zeros(OVERSAMPLING)])
    return torch.as_tensor(k, device=_dev())


def _correction(nx, ny):
    gx = _spheroidal(2.0 * np.abs((np.arange(nx) - nx // 2) / nx))
    gy = _spheroidal(2.0 * np.abs((np.arange(ny) - ny // 2) / ny))
    return torch.as_tensor(np.outer(gx, gy), device=_dev())


def _image_of(grid, sum_weight=None):
    nx, ny = grid.shape[-2:]
    img = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(grid, dim=(-2, -1))),
                             dim=(-2, -1)).real * float(nx * ny) / _correction(nx, ny)
    return img if sum_weight is None else img / sum_weight[..., None, None]


def _tap(table, pos, off):
    return table[(OVERSAMPLING * pos + off).abs()]


def _blocks(d):
    """Time slices of at most about 4M correlations."""
    nt, nb = d.uvw.shape[:2]
    step = max(1, (1 << 22) // max(1, nb * len(d.freq) * d.pols))
    return [(t, min(nt, t + step)) for t in range(0, nt, step)]


def _grid_places(d, t0, t1, margin):
    """Centre cells and distances of the gridder's convention: int(x + 0.5)."""
    got = []
    for k, n in enumerate((d.nx, d.ny)):
        f = torch.as_tensor(d.freq, device=_dev())
        scale = -(f * float(d.incr[k]) * float(n)) / C_LIGHT
        pos = d.uvw[t0:t1, :, k, None] * scale + float(n // 2)
        cell = (pos + 0.5).to(torch.int64)
        got += [pos, cell]
    up, u, vp, v = got
    ok = (u + margin < d.nx) & (v + margin < d.ny) & (u - margin >= 0) & (v - margin >= 0)
    return up, u, vp, v, ok


def _exact_grid(d):
    """grid (planes, pols, nx, ny) and sum of weights of d.vis x d.weight."""
    s, half = d.support, d.support // 2
    table = _kernel(s)
    grid = torch.zeros((d.planes * d.nx * d.ny, d.pols, 2), dtype=torch.float64, device=_dev())
    sw = torch.zeros((d.planes, d.pols), dtype=torch.float64, device=_dev())
    plane = torch.as_tensor(d.chan_map, device=_dev())
    for t0, t1 in _blocks(d):
        up, u, vp, v, ok = _grid_places(d, t0, t1, half)
        ou = torch.floor((u.double() - up) * OVERSAMPLING + 0.5).to(torch.int64)
        ov = torch.floor((v.double() - vp) * OVERSAMPLING + 0.5).to(torch.int64)
        w = d.weight[t0:t1].double()[ok]
        val = torch.view_as_real(d.vis[t0:t1].to(torch.complex128))[ok] * w[..., None]
        base = ((plane.expand_as(u) * d.nx + u) * d.ny + v)[ok]
        ou, ov = ou[ok], ov[ok]
        norm = torch.zeros_like(ou, dtype=torch.float64)
        for i in range(-half, s - half):
            cu = _tap(table, i, ou)
            for j in range(-half, s - half):
                c = cu * _tap(table, j, ov)
                grid.index_add_(0, base + (i * d.ny + j), val * c[:, None, None])
                norm += c
        used = (val != 0).any(dim=-1)
        sw.index_add_(0, plane.expand_as(u)[ok], w * norm[:, None] * used)
    g = torch.view_as_complex(grid).reshape(d.planes, d.nx, d.ny, d.pols)
    return g.permute(0, 3, 1, 2).contiguous(), sw


def _degrid_places(d, t0, t1):
    """Cells and kernel offsets of the degridder's convention: round half to even."""
    got = []
    f = torch.as_tensor(d.freq, device=_dev())
    for k, n in enumerate((d.nx, d.ny)):
        pos = (-float(d.incr[k]) * n * d.uvw[t0:t1, :, k, None]) * f / C_LIGHT + n / 2.0
        cell = torch.round(pos)
        got += [cell.to(torch.int64), torch.round((cell - pos) * OVERSAMPLING).to(torch.int64)]
    x, ox, y, oy = got
    lo = -(d.support // 2)
    hi = lo + d.support - 1
    ok = ((x + lo >= 0) & (x + hi < min(d.nx, d.ny)) & (y + lo >= 0)
          & (y + hi < min(d.nx, d.ny)))
    return x, ox, y, oy, ok


def _exact_degrid(d, model, adjoint_of=None):
    """Model visibilities of the grid `model`, or the transpose applied to adjoint_of."""
    s, half = d.support, d.support // 2
    table = _kernel(s)
    plane = torch.as_tensor(d.chan_map, device=_dev())
    if adjoint_of is None:
        flat = model.permute(0, 2, 3, 1).reshape(-1, d.pols).contiguous()
        out = torch.zeros(tuple(d.uvw.shape[:2]) + (len(d.freq), d.pols), dtype=torch.complex128,
                          device=_dev())
    else:
        out = torch.zeros((d.planes * d.nx * d.ny, d.pols, 2), dtype=torch.float64, device=_dev())
    for t0, t1 in _blocks(d):
        x, ox, y, oy, ok = _degrid_places(d, t0, t1)
        base = ((plane.expand_as(x) * d.nx + x) * d.ny + y)[ok]
        ox, oy = ox[ok], oy[ok]
        wx = [_tap(table, i, ox) for i in range(-half, s - half)]
        wy = [_tap(table, j, oy) for j in range(-half, s - half)]
        norm = sum(wx) * sum(wy)
        if adjoint_of is None:
            acc = torch.zeros((len(base), d.pols), dtype=torch.complex128, device=_dev())
        else:
            val = torch.view_as_real(adjoint_of[t0:t1].to(torch.complex128))[ok]
            val = val / norm[:, None, None]
        for i in range(s):
            for j in range(s):
                c, at = wx[i] * wy[j], base + ((i - half) * d.ny + j - half)
                if adjoint_of is None:
                    acc += flat[at] * c[:, None]
                else:
                    out.index_add_(0, at, val * c[:, None, None])
        if adjoint_of is None:
            block = out[t0:t1]
            block[ok] = acc / norm[:, None]
    if adjoint_of is None:
        return out
    g = torch.view_as_complex(out).reshape(d.planes, d.nx, d.ny, d.pols)
    return g.permute(0, 3, 1, 2).contiguous()


def _exact_weights(d, case):
    chans, pols = case["chans"], case["pols"]
    up, u, vp, v, ok = _grid_places(d, 0, d.uvw.shape[0], 0)
    ok = ok & (up + 0.5 > -1) & (vp + 0.5 > -1)
    w = torch.where(d.flag, torch.full_like(d.weight, float("nan")), d.weight).double()
    w = {1: lambda: w[..., 0], 2: lambda: (w[..., 0] + w[..., 1]) / 2,
         4: lambda: (w[..., 0] + w[..., 3]) / 2}[pols]()
    chan = torch.arange(chans, device=_dev()).expand_as(u)
    counted = ok & ~torch.isnan(w)
    g = torch.zeros(chans * d.nx * d.ny, dtype=torch.float64, device=_dev())
    g.index_add_(0, ((chan * d.nx + u) * d.ny + v)[counted], w[counted])
    # the conjugate of every sample, where it is on the grid
    uc = (-(up - d.nx // 2) + d.nx // 2 + 0.5).to(torch.int64)
    vc = (-(vp - d.ny // 2) + d.ny // 2 + 0.5).to(torch.int64)
    both = counted & (uc >= 0) & (uc < d.nx) & (vc >= 0) & (vc < d.ny)
    g.index_add_(0, ((chan * d.nx + uc) * d.ny + vc)[both], w[both])
    sw = torch.zeros(chans, dtype=torch.float64, device=_dev())
    sw.index_add_(0, chan[counted], 2.0 * w[counted])
    g = g.reshape(chans, 1, d.nx, d.ny)
    r = 5.0 * 10.0 ** -0.5
    f0 = r * r / ((g ** 2).sum(dim=(1, 2, 3)) / sw)
    at = g.reshape(chans, -1)[chan, (u * d.ny + v).clamp(0, d.nx * d.ny - 1)]
    iw = torch.where((at != 0) & (w != 0), w / (f0[chan] * at + 1.0), w)
    iw = torch.where(ok, iw, torch.zeros_like(iw))
    factors = torch.stack([f0, torch.ones_like(f0)]).reshape(2, chans, 1)
    return g, sw.reshape(chans, 1), factors, iw[..., None].expand(-1, -1, -1, pols), None


def _exact_clean(d, case):
    n = case["nx"]
    residual, psf = d.dirty.double(), d.psf.double()
    padded = torch.zeros((2 * n, 2 * n), dtype=torch.float64, device=_dev())
    at = n - n // 2
    padded[at:at + n, at:at + n] = psf  # centre at (n, n)
    model = torch.zeros_like(residual)
    gain, threshold = float(np.float32(0.1)), float(np.float32(1e-4))
    done = 0
    for _ in range(case["iters"]):
        k = int(residual.abs().argmax())
        y, x = divmod(k, n)
        peak = float(residual[y, x])
        if abs(peak) < threshold:
            break
        model[y, x] += gain * peak
        residual -= gain * peak * padded[n - y:2 * n - y, n - x:2 * n - x]
        done += 1
    return model, residual, None, float(residual.abs().max()), float(model.abs().sum())


def _exact_mosaic(d, case):
    cf = (d.cf * d.gradient[0]).contiguous()
    reach = int(d.support.max())
    up, u, vp, v, ok = _grid_places(d, 0, d.uvw.shape[0], reach)
    n = cf.shape[-1]
    ou = torch.floor((u.double() - up) * MOSAIC_OS + 0.5).to(torch.int64)[ok] + n // 2
    ov = torch.floor((v.double() - vp) * MOSAIC_OS + 0.5).to(torch.int64)[ok] + n // 2
    chan = torch.arange(d.planes, device=_dev()).expand_as(u)[ok]
    which = torch.as_tensor(d.cfb, device=_dev())[None, :, None].expand_as(u)[ok]
    cfc = torch.as_tensor(d.cfc, device=_dev())[chan]
    sup = torch.as_tensor(d.support, device=_dev())[which, cfc, 0, 0]
    w = d.weight[ok]
    val = d.vis[ok] * w
    base = (chan * d.nx + u[ok]) * d.ny + v[ok]
    first = (which * cf.shape[1] + cfc) * n * n
    grid = torch.zeros((d.planes * d.nx * d.ny, d.pols, 2), dtype=torch.float64, device=_dev())
    norm = torch.zeros(len(base), dtype=torch.complex128, device=_dev())
    flat = cf.reshape(-1)
    half = reach // 2
    for i in range(-half, reach - half):
        for j in range(-half, reach - half):
            fu, fv = MOSAIC_OS * i + ou, MOSAIC_OS * j + ov
            inside = ((fu >= 0) & (fu < n) & (fv >= 0) & (fv < n) & (i >= -(sup // 2))
                      & (i < sup - sup // 2) & (j >= -(sup // 2)) & (j < sup - sup // 2))
            c = torch.where(inside, flat[torch.where(inside, first + fu * n + fv, 0)], 0)
            grid.index_add_(0, base + (i * d.ny + j), torch.view_as_real(val * c[:, None]))
            norm += c
    sw = torch.zeros((d.planes, d.pols), dtype=torch.float64, device=_dev())
    sw.index_add_(0, chan, w * (norm ** 2).real[:, None])
    g = torch.view_as_complex(grid).reshape(d.planes, d.nx, d.ny, d.pols)
    return g.permute(0, 3, 1, 2).contiguous(), sw


def exact(case, seed):
    kind = case["kind"]
    if kind == "loop":
        return None  # the controller's decisions have no short restatement
    d = _inputs(case, seed)
    if kind == "image":
        return _image_of(d.grid, d.sum_weight)
    if kind == "clean":
        return _exact_clean(d, case)
    d.nx, d.ny, d.pols = case["nx"], case["ny"], case.get("pols", 1)
    d.support = d.support if kind == "mosaic" else case.get("support", 7)
    cube = case.get("cube", False) or kind in ("mosaic", "batched")
    d.planes = case["chans"] if cube else 1
    d.chan_map = np.arange(case["chans"]) if cube else np.zeros(case["chans"], dtype=int)
    if kind == "weights":
        return _exact_weights(d, case)
    if kind == "mosaic":
        return _exact_mosaic(d, case)
    if kind == "forward":
        sky = d.sky.double()
        predicted = _exact_degrid(d, _centred_fft(sky / _correction(d.nx, d.ny)))
        back = (predicted.to(torch.complex64) - d.vis).to(torch.complex128)
        return predicted, _image_of(_exact_degrid(d, None, back))
    if kind == "batched":
        return _exact_grid(d)
    if kind == "double":
        return _exact_grid(d) + (_exact_degrid(d, d.model),)
    grid, sum_weight = _exact_grid(d)
    model = _centred_fft(d.sky)
    predicted = _exact_degrid(d, model)
    if kind == "cycle":
        return grid, sum_weight, predicted
    predicted = torch.where(d.flag, torch.zeros_like(predicted), predicted)
    return _image_of(grid, sum_weight), sum_weight, predicted, d.vis - predicted
