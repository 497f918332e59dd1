"""The FP32 degridder's store mode against its accumulating mode on zeroed
values: the same FP32 sums of taps, scaled by 1 / norm in FP64 and rounded
once, so no component differs by more than one FP32 ulp (1.2e-7 of it; the
reciprocal is formed from two factors in one and from their product in the
other)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npol,flagged", [(1, False), (1, True), (2, False), (2, True), (3, False),
                                          (4, True)])
@pytest.mark.parametrize("support", [3, 6, 7, 9])
def test_store_scales_in_double_precision(npol, flagged, support):
    from astroviper_b200.gridder import Gridder
    rng = np.random.default_rng(npol + 10 * support)
    nt, nb, nchan, nx, ny = 23, 37, 3, 128, 150
    cell = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8
    uvw = rng.normal(size=(nt, nb, 3)) * 500.0
    G = Gridder(uvw, np.array([1.4e9, 1.5e9, 1.6e9]), (nx, ny), cell, npol, support=support)
    grid = torch.as_tensor(rng.normal(size=(1, npol, nx, ny))
                           + 1j * rng.normal(size=(1, npol, nx, ny)), device="cuda")
    flag = None
    if flagged:
        flag = torch.as_tensor(rng.uniform(size=(nt, nb, nchan, npol)) < 0.2, device="cuda")
    stored = torch.view_as_real(G.degrid(grid, flag=flag))
    zeros = torch.zeros((nt, nb, nchan, npol), dtype=torch.complex64, device="cuda")
    added = torch.view_as_real(G.degrid(grid, zeros, flag=flag, accumulate=True))
    assert added.abs().max() > 0
    assert bool(((stored - added).abs() <= 1.2e-7 * added.abs()).all())
