"""Gridder.plan() then degrid() on odd image sizes: the degridder's centre is
n / 2, not the gridder's cell n // 2, so a plan shared with the gridder would
degrid half a cell off.  Against the plain FP64 degridder, within the FP32
path's rounding (1e-5 of the largest sample; half a cell is of order 1)."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(128, 96), (127, 96), (128, 97), (127, 97)])
@pytest.mark.parametrize("mode", ["continuum", "cube"])
def test_planned_degrid(nx, ny, mode):
    from astroviper_b200 import _kernels as K
    from astroviper_b200.gridder import Gridder
    rng = np.random.default_rng(nx + ny)
    cell = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8
    nt, nb, nchan, npol = 3, 40, 2, 2
    uvw = rng.normal(size=(nt, nb, 3)) * 500.0
    freq = np.array([1.4e9, 1.5e9])
    G = Gridder(uvw, freq, (nx, ny), cell, npol, support=7, chan_mode=mode)
    G.plan()
    n_img = nchan if mode == "cube" else 1
    grid = torch.as_tensor(rng.normal(size=(n_img, npol, nx, ny))
                           + 1j * rng.normal(size=(n_img, npol, nx, ny)), device="cuda")
    got = G.degrid(grid).to(torch.complex128)
    cmap = (np.arange(nchan) / nchan * n_img).astype(int)
    ref = K.degrid(grid, uvw, freq, (-cell[0] * nx, -cell[1] * ny), (nx / 2, ny / 2), cmap,
                   np.arange(npol), O.create_prolate_spheroidal_kernel_1D(100, 7), 7, 100,
                   nvchan=nchan, nvpol=npol, precision="fp64")
    assert (got - ref).abs().max() <= 1e-5 * ref.abs().max()
