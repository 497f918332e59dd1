"""Minimum and maximum of images whose extreme is a zero: its sign is the
image's, over one block and over many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 40, 700])
def test_sign_of_a_zero_extreme(dtype, n):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(n)
    img = rng.uniform(0.5, 1.0, (n, n)).astype(dtype)
    for zero in (-0.0, 0.0):
        low = -img
        low[rng.uniform(size=low.shape) < 0.3] = zero
        low[0, 0] = zero
        assert str(K.maximg(low).cpu().numpy()[1]) == str(dtype(zero))
        high = img.copy()
        high[rng.uniform(size=high.shape) < 0.3] = zero
        high[-1, -1] = zero
        assert str(K.maximg(high).cpu().numpy()[0]) == str(dtype(zero))
