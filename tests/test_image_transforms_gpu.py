"""Grid -> image and image -> grid through the real transforms, against numpy.

Sizes cover odd and even axes, single rows and columns, and the edges of the
kernels' blocks (128 columns, 32 rows, 4 rows in flight).  Both sides are FP64
transforms of n points, whose norm-wise error is about eps log2(n) (eps =
1.1e-16, below 3e-15 here); the grid correction divides by at least 4e-3
squared at the corners, so an image may be off by up to 1e-10 of its norm."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 6), (7, 1), (2, 3), (5, 4), (31, 33), (32, 128), (33, 129), (36, 127),
         (64, 257), (130, 255)]


def _rel(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


def _centred(x, f):
    return np.fft.fftshift(f(np.fft.ifftshift(x, axes=(-2, -1)), axes=(-2, -1)), axes=(-2, -1))


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("planes", [1, 3])
def test_grid_to_image_is_the_real_part_of_the_complex_transform(nx, ny, planes):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(nx * 1000 + ny)
    g = rng.normal(size=(planes, nx, ny)) + 1j * rng.normal(size=(planes, nx, ny))
    sw = rng.uniform(1.0, 2.0, planes)
    ref = _centred(g, np.fft.ifft2).real * nx * ny
    got = K.grid_to_image(g, apply_corr=False).cpu().numpy()
    assert _rel(got, ref) <= 1e-14
    got = K.grid_to_image(g, sw, apply_corr=False, out_dtype=torch.float32).cpu().numpy()
    assert _rel(got, ref / sw[:, None, None]) <= 1e-7
    got = K.grid_to_image(g.astype(np.complex64), sw, apply_corr=False).cpu().numpy()
    assert _rel(got, ref / sw[:, None, None]) <= 1e-6
    corr = K.corr_term(nx, ny).cpu().numpy()
    ok = corr != 0
    got = K.grid_to_image(g, sw).cpu().numpy()
    assert _rel(got[:, ok], (ref / corr / sw[:, None, None])[:, ok]) <= 1e-10


@pytest.mark.parametrize("nx,ny", SIZES)
def test_real_image_forward_transform(nx, ny):
    from astroviper_b200 import _kernels as K
    from astroviper_b200.core.imaging.fft import fft_lm_to_uv
    rng = np.random.default_rng(nx * 1000 + ny)
    x = rng.normal(size=(2, nx, ny))
    ref = _centred(x, np.fft.fft2)
    assert _rel(K.fft_shifted(x, inverse=False).cpu().numpy(), ref) <= 1e-14
    assert _rel(fft_lm_to_uv(x, [1, 2]), ref) <= 1e-14
    assert _rel(fft_lm_to_uv(x.transpose(1, 2, 0), [0, 1]), ref.transpose(1, 2, 0)) <= 1e-14
    assert fft_lm_to_uv((10 * x).astype(np.int64), [1, 2]).dtype == np.complex128
    assert fft_lm_to_uv(x.astype(np.float32), [1, 2]).dtype == np.complex64


@pytest.mark.parametrize("planes", [2367, 4735, 4737, 5000])
def test_many_planes_take_a_block_for_two(planes):
    """Around the number of blocks from which a block takes two planes (16 per
    SM of 148), even and odd: each plane is the one of a call by itself."""
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(planes)
    g = rng.normal(size=(planes, 5, 4)) + 1j * rng.normal(size=(planes, 5, 4))
    sw = rng.uniform(1.0, 2.0, planes)
    got = K.grid_to_image(g, sw, apply_corr=False).cpu().numpy()
    ref = _centred(g, np.fft.ifft2).real * 20 / sw[:, None, None]
    assert np.abs(got - ref).max() <= 1e-14 * np.abs(ref).max()
    one = K.grid_to_image(g[-1:], sw[-1:]).cpu().numpy()
    assert np.abs(K.grid_to_image(g, sw).cpu().numpy()[-1:] - one).max() <= 1e-14 * np.abs(one).max()
