"""The binned FP64 gridder and degridder against the plain FP64 kernels, over
every form that the plain ones accept and the binned ones take: supports,
polarisation counts and maps, input types, flags, phases, dropped channels,
NaN, zero and infinite data, grids in either precision, sizes from one sample.

Both gridders add the same FP64 products in another order, so a cell differs
by rounding alone: 1e-13 of the largest cell covers sums of the few thousand
samples here (eps x terms = 1.1e-16 x 1e3).  The degridders are bit-identical."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def both(monkeypatch):
    from astroviper_b200 import _kernels as K

    def run(f, *a, **kw):
        out = []
        for binned in (False, True):
            monkeypatch.setattr(K, "_binning_pays", lambda *x, b=binned: b)
            n0 = K.lib().av_launch_count()
            out.append(f(*a, **kw))
            # a plan is several launches, the plain kernel one
            assert (K.lib().av_launch_count() - n0 > 3) == binned
        return out

    return run


def _data(rng, nt, nb, nchan, npol, vdt, wdt):
    uvw = rng.normal(size=(nt, nb, 3)) * 900.0
    uvw[0, 0, 0] = np.nan
    vis = (rng.normal(size=(nt, nb, nchan, npol))
           + 1j * rng.normal(size=(nt, nb, nchan, npol))).astype(vdt)
    wt = rng.uniform(0.2, 2.0, (nt, nb, nchan, npol)).astype(wdt)
    wt[rng.uniform(size=wt.shape) < 0.1] = 0.0
    vis[rng.uniform(size=vis.shape) < 0.05] = np.nan
    return uvw, vis, wt


def _close(a, b):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    ok = np.isfinite(a)
    tol = 1e-13 if a.dtype in (np.complex128, np.float64) else 1e-6
    assert np.abs(a[ok] - b[ok]).max() <= tol * max(np.abs(b[ok]).max(), 1e-300)


CELL = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8


@pytest.mark.parametrize("support", [3, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("npol,pol_map", [(1, [0]), (2, [1, 0]), (3, [0, -1, 1]), (4, [3, 3, 0, 1])])
@pytest.mark.parametrize("vdt,wdt", [(np.complex128, np.float64), (np.complex64, np.float64),
                                     (np.complex128, np.float32)])
def test_grid(both, support, npol, pol_map, vdt, wdt):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(support * 10 + npol)
    uvw, vis, wt = _data(rng, 37, 5, 3, npol, vdt, wdt)
    freq = np.array([1.0e9, 1.2e9, 1.3e9])
    for chan_map, do_psf, os_ in (([0, 1, 0], False, 100), ([0, 5, -1], True, 37)):
        cgk = K.pswf_table(os_, support)
        args = (vis, torch.as_tensor(wt), uvw, freq, np.array(chan_map), np.array(pol_map), cgk,
                (61, 44), CELL, support, os_, 2, 4)
        (g0, s0), (g1, s1) = both(K.grid, *args, do_psf=do_psf, precision="fp64")
        assert g0.abs().nan_to_num().max() > 0
        _close(g1, g0)
        _close(s1, s0)


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 33, 1), (65, 1, 2), (64, 16, 4)])
def test_grid_sizes_infinities_and_single_precision_grids(both, shape):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(sum(shape))
    uvw, vis, wt = _data(rng, *shape, 2, np.complex128, np.float64)
    if shape != (1, 1, 1):
        vis[0, -1, 0, 1] = np.inf
    freq = np.linspace(1.0e9, 1.1e9, shape[2])
    cgk = K.pswf_table(100, 7)
    for dt in (torch.complex128, torch.complex64):
        def f():
            g = torch.full((1, 2, 48, 50), 0.5 + 0.25j, dtype=dt, device="cuda")
            return K.grid(vis, torch.as_tensor(wt), uvw, freq, np.zeros(shape[2], int),
                          np.arange(2), cgk, (48, 50), CELL, 7, 100, 1, 2, grid_out=g,
                          precision="fp64")
        (g0, s0), (g1, s1) = both(f)
        _close(g1, g0)
        _close(s1, s0)


@pytest.mark.parametrize("support", [3, 4, 5, 6, 7, 8, 9])
@pytest.mark.parametrize("nvpol,g_npol", [(1, 1), (2, 3), (3, 2), (4, 4)])
@pytest.mark.parametrize("gdt,vdt", [(np.complex128, np.complex128), (np.complex64, np.complex64)])
def test_degrid_bit_identical(both, support, nvpol, g_npol, gdt, vdt):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(support * 100 + nvpol)
    nt, nb, nc, n2, n3 = 41, 4, 3, 57, 70
    uvw = rng.normal(size=(nt, nb, 3)) * 900.0
    uvw[1, 1, 1] = np.nan
    freq = np.array([1.0e9, 1.2e9, 1.3e9])
    g = rng.normal(size=(2, g_npol, n2, n3)) + 1j * rng.normal(size=(2, g_npol, n2, n3))
    g = g.astype(gdt)
    v0 = (rng.normal(size=(nt, nb, nc, nvpol)) + 0j).astype(vdt)
    flag = rng.uniform(size=v0.shape) < 0.1
    dph = rng.normal(size=(nt, nb))
    scale, off = (-CELL[0] * n2, -CELL[1] * n3), (n2 / 2, n3 / 2)
    for cm, pm, fl, dp, os_ in (([0, 1, 0], np.arange(nvpol) % g_npol, None, None, 100),
                                ([1, -1, 2], np.arange(nvpol)[::-1] - (nvpol > 1), flag, dph, 63)):
        cf = K.pswf_table(os_, support)

        def f():
            return K.degrid(g, uvw, freq, scale, off, np.array(cm), np.array(pm), cf, support,
                            os_, values=torch.as_tensor(v0).cuda(), flag=fl, dphase=dp,
                            precision="fp64")
        a, b = both(f)
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
        assert not torch.equal(a, torch.as_tensor(v0).cuda())


def test_rule_prefers_the_plain_kernels_for_small_calls():
    from astroviper_b200 import _kernels as K
    assert not K._binning_pays(33.0, 100, 2, 1, 512, 512, 7)
    assert K._binning_pays(33.0, 100_000, 2, 1, 512, 512, 7)
    assert not K._binning_pays(33.0, 100_000, 2, 1, 512, 512, 10)
    assert not K._binning_pays(33.0, 1 << 31, 2, 1, 512, 512, 7)
    assert not K._binning_pays(2.5, 100_000, 2, 4096, 512, 512, 7)
