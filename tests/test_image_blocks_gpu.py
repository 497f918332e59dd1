"""The image passes at the edges of their blocks (128 columns, 16 rows, 8 rows
in flight), against numpy with the bounds of test_image_transforms_gpu."""
import numpy as np
import pytest
from test_image_transforms_gpu import _centred, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [127, 128, 129, 256])
@pytest.mark.parametrize("nx", [7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33])
def test_block_edges(nx, ny):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(nx * 1000 + ny)
    g = rng.normal(size=(3, nx, ny)) + 1j * rng.normal(size=(3, nx, ny))
    sw = rng.uniform(1.0, 2.0, 3)
    ref = _centred(g, np.fft.ifft2).real * nx * ny
    assert _rel(K.grid_to_image(g, sw, apply_corr=False).cpu().numpy(),
                ref / sw[:, None, None]) <= 1e-14
    corr = K.corr_term(nx, ny).cpu().numpy()
    got = K.grid_to_image(g, sw).cpu().numpy()
    assert _rel(got, ref / corr / sw[:, None, None]) <= 1e-10
    x = rng.normal(size=(3, nx, ny))
    assert _rel(K.fft_shifted(x, inverse=False).cpu().numpy(), _centred(x, np.fft.fft2)) <= 1e-14
