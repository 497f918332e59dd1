"""The order in which the persistent gridders and degridders take a plan's
chunks of records (a plane's outer chunks first, plane by plane in turn): every
chunk is taken once, whatever the numbers of planes and chunks.  The oracle is
linearity: each time step alone is one chunk, and their sum is the whole call.

The grids are FP64 sums of the same products in another order (1e-13 of the
largest cell covers the 3e4 terms here: eps x sqrt(terms) = 2e-14); a degridded
sample is the same FP32 or TF32 sum in either call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npol", [1, 2, 4])
@pytest.mark.parametrize("nt,nb,planes", [(1, 700, 1), (41, 700, 1), (40, 250, 3), (40, 190, 4),
                                          (31, 20, 33), (80, 23, 33), (60, 6, 128)])
def test_each_chunk_once(npol, nt, nb, planes):
    from astroviper_b200.gridder import Gridder
    rng = np.random.default_rng(nt * nb + planes + npol)
    cell = np.array([-2.0, 2.0]) * np.pi / 180 / 3600 * 8
    uvw = rng.normal(size=(nt, nb, 3)) * 700.0
    freq = 1.4e9 + 1e6 * np.arange(planes)
    shape = (nt, nb, planes, npol)
    vis = torch.as_tensor((rng.normal(size=shape) + 1j * rng.normal(size=shape))
                          .astype(np.complex64), device="cuda")
    wt = torch.as_tensor(rng.uniform(0.5, 1.5, shape).astype(np.float32), device="cuda")

    def make(t):
        return Gridder(uvw[t], freq, (192, 160), cell, npol, support=7,
                       chan_mode="cube" if planes > 1 else "continuum")

    whole = make(slice(None))
    grid, sw = whole.grid(vis, wt)
    parts = [make(slice(t, t + 1)) for t in range(nt)]
    g1, s1 = torch.zeros_like(grid), torch.zeros_like(sw)
    for t, p in enumerate(parts):
        g, s = p.grid(vis[t:t + 1], wt[t:t + 1])
        g1 += g
        s1 += s
    assert (grid - g1).abs().max() <= 1e-13 * g1.abs().max()
    assert (sw - s1).abs().max() <= 1e-13 * s1.abs().max()

    model = torch.randn(grid.shape, dtype=torch.complex128, device="cuda")
    out = torch.full(shape, float("nan"), dtype=torch.complex64, device="cuda")
    whole.degrid(model, out)
    for t, p in enumerate(parts):
        one = torch.full((1,) + shape[1:], float("nan"), dtype=torch.complex64, device="cuda")
        p.degrid(model, one)
        assert torch.equal(out[t:t + 1], one)
