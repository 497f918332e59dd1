"""A degridder's kernel table whose taps at offset 0 add up to exactly zero in
FP64 but not when each is rounded to FP32: samples there have no norm, so they
are written as zeros and left alone when accumulating."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npol", [1, 2])
def test_taps_that_cancel(npol):
    from astroviper_b200.gridder import C_LIGHT, Gridder
    n, os_ = 64, 10
    rng = np.random.default_rng(npol)
    taps = rng.uniform(0.5, 1.0, 3 * os_)
    taps[[0, os_, 2 * os_]] = -2.0321471219535843, 0.6732655185893088, 0.3428080423874833
    at_0 = taps[[2 * os_, os_, 0, os_, 2 * os_]]
    assert np.cumsum(at_0)[-1] == 0.0
    assert np.cumsum(at_0.astype(np.float32).astype(np.float64))[-1] != 0.0
    uvw = rng.integers(-20, 20, (6, 7, 3)).astype(np.float64)
    uvw[::2, ::2, :2] += 0.3  # the other samples sit on a cell in u and v
    uvw[1, 1, 0] += 0.3       # and this one in v only
    G = Gridder(uvw, np.array([C_LIGHT]), (n, n), (-1.0 / n, 1.0 / n), npol, support=5,
                oversampling=os_)
    G.cgk = torch.as_tensor(taps, device="cuda")
    grid = torch.as_tensor(rng.normal(size=(1, npol, n, n)) + 1j, device="cuda")
    off = np.zeros((6, 7), dtype=bool)
    off[::2, ::2] = True
    stored = G.degrid(grid).cpu().numpy()[:, :, 0]
    assert np.all(stored[~off] == 0) and np.all(stored[off] != 0)
    ones = torch.ones((6, 7, 1, npol), dtype=torch.complex64, device="cuda")
    added = G.degrid(grid, ones, accumulate=True).cpu().numpy()[:, :, 0]
    assert np.all(added[~off] == 1) and np.all(added[off] != 1)
