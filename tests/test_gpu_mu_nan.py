"""The chemical potential at T = 0 of device bands with NaN among them."""
import numpy as np
import pytest

from test_gpu_mu import device_mu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(4, 9), (16, 700)])
@pytest.mark.parametrize("share", [0.1, 0.6])
def test_nan_values_are_not_counted(lqm, ctx, n, nk, share):
    """The k-th value is the k-th of the numbers, and their largest where there are fewer."""
    rng = np.random.default_rng(n)
    bands = rng.normal(size=(n, nk))
    bands[rng.random((n, nk)) < share] = np.nan
    v = np.sort(bands[np.isfinite(bands)])
    for filling in (0.05, 0.3, 0.5, 0.9, 0.999):
        i = int(np.floor(filling * (n * nk - 1)))
        want = (v[min(i, v.size - 1)] + v[min(i + 1, v.size - 1)]) / 2
        assert device_mu(lqm, ctx, bands, filling, 0.0) == want, filling
