"""The workspace sizes of the image transforms: each direction runs in its own
size, and the common size covers both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,nx,ny", [(1, 1, 1), (2, 7, 6), (1, 33, 129), (3, 64, 61),
                                          (1, 509, 260)])
def test_each_direction_runs_in_its_size(planes, nx, ny):
    from astroviper_b200 import _kernels as K
    from astroviper_b200._lib import AV_C128, AV_F64, AV_OK, lib
    both = lib().av_grid_to_image_workspace_size(planes, nx, ny)
    inv = lib().av_real_fft_workspace_size(planes, nx, ny, 1)
    fwd = lib().av_real_fft_workspace_size(planes, nx, ny, 0)
    assert both == max(inv, fwd) and min(inv, fwd) > 0
    g = torch.randn((planes, nx, ny), dtype=torch.complex128, device="cuda")
    x = torch.empty((planes, nx, ny), dtype=torch.float64, device="cuda")
    _b, ptr, _n = K.workspace(inv)
    assert lib().av_grid_to_image(K.p(g), AV_C128, None, K.p(x), AV_F64, planes, nx, ny, 0, ptr,
                                  inv, K.stream_ptr()) == AV_OK
    assert torch.equal(x, K.grid_to_image(g, apply_corr=False))
    h = torch.empty_like(g)
    _b, ptr, _n = K.workspace(fwd)
    assert lib().av_image_to_grid(K.p(x), AV_F64, K.p(h), AV_C128, planes, nx, ny, 0, ptr, fwd,
                                  K.stream_ptr()) == AV_OK
    assert torch.equal(h, K.fft_shifted(x, inverse=False))
