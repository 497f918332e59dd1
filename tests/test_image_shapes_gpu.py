"""The image passes in each of their block shapes (eight row groups side by
side up to 64 columns, 4 rows to a block where blocks are few, 16 else), at
the edges of the groups, against numpy with the bounds of
test_image_transforms_gpu."""
import numpy as np
import pytest
from test_image_transforms_gpu import _centred, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,nx,ny", [
    (2, nx, ny) for nx in (1, 3, 4, 5, 31, 32, 33, 70) for ny in (2, 15, 16, 17, 64, 65, 130)
] + [(60, nx, 129) for nx in (31, 32, 33)] + [(300, 17, 40), (3, 1000, 3)])
def test_block_shapes(planes, nx, ny):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(nx * 1000 + ny)
    g = rng.normal(size=(planes, nx, ny)) + 1j * rng.normal(size=(planes, nx, ny))
    sw = rng.uniform(1.0, 2.0, planes)
    ref = _centred(g, np.fft.ifft2).real * nx * ny / sw[:, None, None]
    assert _rel(K.grid_to_image(g, sw, apply_corr=False).cpu().numpy(), ref) <= 1e-14
    corr = K.corr_term(nx, ny).cpu().numpy()
    assert _rel(K.grid_to_image(g, sw).cpu().numpy(), ref / corr) <= 1e-10
    x = rng.normal(size=(planes, nx, ny))
    assert _rel(K.fft_shifted(x, inverse=False).cpu().numpy(), _centred(x, np.fft.fft2)) <= 1e-14
