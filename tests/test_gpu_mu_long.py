"""The chemical-potential search at T > 0 around the list length from which a pass over the
values takes one bisection step instead of three (2048 values per SM)."""
import numpy as np
import pytest

from oracle import kspace as K
from test_gpu_mu import device_mu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1, 2 ** 20])
def test_long_lists_match_oracle(lqm, ctx, extra):
    """Both are roots of the same filling to its rounding: mu agrees to 1e-10 over a filling
    that rises (as the shorter lists of test_gpu_mu)."""
    import torch
    nv = 2048 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    n = next(d for d in (16, 5, 3, 1) if nv % d == 0)
    rng = np.random.default_rng(nv)
    bands = np.sort(rng.normal(size=(n, nv // n)), axis=0)
    w = rng.uniform(0.5, 1.5, nv // n)
    w /= w.sum()
    for filling, T, ww in ((0.2, 0.05, None), (0.77, 0.01, None), (0.4, 0.1, w)):
        mu, ref = device_mu(lqm, ctx, bands, filling, T, ww), K.chemicalpotential(bands, filling, T, ww)
        assert abs(mu - ref) <= 1e-10 * max(1.0, abs(ref)), filling
    with pytest.raises(lqm.LQMError):
        device_mu(lqm, ctx, bands, 1.5, 0.01)
