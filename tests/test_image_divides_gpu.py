"""The image passes' divides (by the sum of weights and by the grid correction)
against IEEE divides of the undivided image.  The sum's reciprocal is rounded,
so by Markstein's theorem its quotient is the divide's to the last bit, and the
zeros, infinities, NaN and extremes go through a divide; the correction's
reciprocal comes from a Newton step, within one ulp."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SUMS = [1.0, 3.0, 0.7, 1.0 / 3.0, -2.5e4, 123456.789, 1e-300, 1e300, 1e-20, 1e-21, 1e-100, 5e-324,
        1.7976931348623157e308, 0.0, -0.0, np.inf, -np.inf, np.nan, 2.0 ** -1022, 2.0 - 2.0 ** -52]


def _same_bits(a, b):
    """Equal bits, any NaN for any NaN."""
    nan = torch.isnan(a) & torch.isnan(b)
    return bool(((a.view(torch.int64) == b.view(torch.int64)) | nan).all())


@pytest.mark.parametrize("scale", [1.0, 1e-150, 1e-290, 1e-307, 1e240, 1e300])
@pytest.mark.parametrize("nx,ny", [(33, 130), (64, 64)])
def test_sum_of_weights(scale, nx, ny):
    from astroviper_b200 import _kernels as K
    g = torch.Generator("cuda").manual_seed(nx)
    grid = torch.randn((len(SUMS), nx, ny), generator=g, dtype=torch.complex128, device="cuda")
    grid *= scale
    grid[2] = 0.0
    sw = torch.tensor(SUMS, dtype=torch.float64, device="cuda")
    image = K.grid_to_image(grid, apply_corr=False)
    assert _same_bits(K.grid_to_image(grid, sw, apply_corr=False), image / sw[:, None, None])
    got = K.grid_to_image(grid, sw, apply_corr=False, out_dtype=torch.float32)
    want = (image / sw[:, None, None]).float()
    assert bool(((got == want) | (torch.isnan(got) & torch.isnan(want))).all())


@pytest.mark.parametrize("what", ["random", "zero", "inf", "nan", "tiny", "huge"])
@pytest.mark.parametrize("nx,ny", [(33, 130), (512, 384), (1, 1), (7, 2)])
def test_grid_correction(what, nx, ny):
    from astroviper_b200 import _kernels as K
    g = torch.Generator("cuda").manual_seed(nx)
    grid = torch.randn((2, nx, ny), generator=g, dtype=torch.complex128, device="cuda")
    if what == "zero":
        grid[0] = 0.0
    elif what in ("inf", "nan"):
        grid[1, nx // 2, ny // 3] = float(what)
    elif what in ("tiny", "huge"):
        grid *= 1e-300 if what == "tiny" else 1e300
    corr = K.corr_term(nx, ny)
    want = K.grid_to_image(grid, apply_corr=False) / corr
    got = K.grid_to_image(grid, apply_corr=True)
    finite = torch.isfinite(want)
    assert bool((finite == torch.isfinite(got)).all())
    assert bool((torch.isnan(want) == torch.isnan(got)).all())
    ulp = 2.0 ** -52 * want.abs().clamp(min=2.0 ** -1022)
    assert bool(((got - want).abs() <= ulp)[finite].all())
