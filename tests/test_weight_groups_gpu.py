"""The weight kernels at the edges of their groups of 16 channels and of their
blocks of 256 threads (blocks that hold the ends of several groups, one series
spread over many threads), with the restatement of test_weight_walk_gpu and,
like there, sums that are exact."""
import numpy as np
import pytest
import torch
from test_weight_walk_gpu import CELL, _restate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nb,nchan", [(1, 1, 300), (1, 2, 33), (3, 1, 16), (3, 1, 17),
                                         (2, 16, 16), (1, 17, 31), (3000, 1, 1), (517, 2, 3)])
def test_groups_of_channels(nt, nb, nchan):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(nt + 10 * nb + 100 * nchan)
    n = (64, 41)
    uvw = np.cumsum(rng.normal(size=(nt, nb, 3)) * 20.0, axis=0) + rng.normal(size=(nb, 3)) * 300
    freq = np.linspace(1.0e9, 1.4e9, nchan)
    wt = rng.integers(0, 128, (nt, nb, nchan, 1)) / 64.0
    g, sw, places = _restate(uvw, freq, wt[..., 0], n, CELL)
    gd, sd = K.weight_density(uvw, freq, wt, None, n, CELL)
    assert np.array_equal(gd.cpu().numpy(), g)
    assert np.array_equal(sd.cpu().numpy(), sw)
    fac = np.array([rng.uniform(0.5, 2.0, (nchan, 1)), np.ones((nchan, 1))])
    iw, err = K.briggs_apply(gd, fac, uvw, freq, wt, None, n, CELL, out_dtype=torch.float64)
    ref = np.zeros(wt.shape[:3])
    on = places[..., 0] >= 0
    _, _, c = np.nonzero(on)
    dens = g[c, 0, places[on][:, 0], places[on][:, 1]]
    ref[on] = wt[on][:, 0] / np.where(dens == 0, 1.0, fac[0, c, 0] * dens + fac[1, c, 0])
    assert int(err.item()) == 0
    assert np.array_equal(iw.cpu().numpy()[..., 0], ref)
