"""The FP32 degridder's store mode (complex64, up to 4 polarisations, no phase)
over the forms its stores and flag reads branch on: the polarisation count,
flags or none, and values and flags that start off the widest alignment.
Against the plain FP64 degridder within the FP32 path's bound (1e-6 of the
largest value); flagged and skipped samples are exact zeros."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npol", [1, 2, 3, 4])
@pytest.mark.parametrize("flagged", [False, True])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("support", [3, 7, 9])
def test_store(npol, flagged, off, support):
    from astroviper_b200 import _kernels as K
    from astroviper_b200.gridder import Gridder
    rng = np.random.default_rng(npol + 10 * support)
    n = 128
    cell = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8
    nt, nb, nchan = 5, 37, 3
    uvw = rng.normal(size=(nt, nb, 3)) * 500.0
    uvw[0, 0, 0] = np.nan  # skipped
    freq = np.array([1.4e9, 1.5e9, 1.6e9])
    shape = (nt, nb, nchan, npol)
    size = int(np.prod(shape))
    G = Gridder(uvw, freq, (n, n), cell, npol, support=support)
    grid = torch.as_tensor(rng.normal(size=(1, npol, n, n)) + 1j * rng.normal(size=(1, npol, n, n)),
                           device="cuda")
    values = torch.full((size + 1,), float("nan"), dtype=torch.complex64, device="cuda")
    values = values[off:off + size].view(shape)
    flag = None
    if flagged:
        f = torch.as_tensor(rng.uniform(size=size + 1) < 0.3, device="cuda")
        flag = f[off:off + size].view(shape)
    got = G.degrid(grid, values, flag=flag).to(torch.complex128)
    ref = K.degrid(grid, uvw, freq, (-cell[0] * n, -cell[1] * n), (n / 2, n / 2), np.zeros(nchan, int),
                   np.arange(npol), O.create_prolate_spheroidal_kernel_1D(100, support), support, 100,
                   nvchan=nchan, nvpol=npol, precision="fp64")
    ref[0, 0] = 0.0
    if flagged:
        ref[flag] = 0.0
        assert (got[flag] == 0).all()
    assert (got[0, 0] == 0).all()
    assert (got - ref).abs().max() <= 1e-6 * ref.abs().max()
