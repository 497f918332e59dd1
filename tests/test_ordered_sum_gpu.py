"""The ordered sum of |x| against the same sequential sum on the host, equal to
the last bit, for arrays on both sides of the largest grid (1024 blocks of
16384 elements): a few thousand non-zeros with the first, the last and both
sides of the blocks' borders among them, magnitudes whose sum depends on the
order, NaN and zeros of both signs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16385, 1024 * 16384 - 1, 1024 * 16384, 1024 * 16384 + 1, 20_000_003])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_sum(n, dt):
    from astroviper_b200 import _kernels as K
    rng = np.random.default_rng(n)
    blocks = min(-(-n // 16384), 1024)
    per = -(-n // blocks)
    edges = np.arange(0, n, per)[:: max(1, blocks // 300)]
    at = np.concatenate([edges, edges[1:] - 1, [n - 1], rng.integers(0, n, 2000)])
    at = np.unique(at)
    x = np.zeros(n, dt)
    x[at] = (rng.normal(size=at.size) * 10.0 ** rng.uniform(-6, 6, at.size)).astype(dt)
    x[1:n:n // 7][x[1:n:n // 7] == 0] = -0.0

    def expected():
        s = dt(0)
        for v in np.abs(x[at]):
            s = dt(s + v)
        return s
    assert K.abs_sum_ordered(x[None]).cpu().numpy()[0] == expected()
    x[at[len(at) // 2]] = np.nan
    assert np.isnan(K.abs_sum_ordered(x[None]).cpu().numpy()[0])
