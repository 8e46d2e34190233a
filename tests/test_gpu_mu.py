"""The chemical-potential search on the device (one cooperative launch) at the sizes where
its split of the values changes."""
import ctypes

import numpy as np
import pytest

from oracle import kspace as K

pytestmark = pytest.mark.gpu


def device_mu(lqm, ctx, bands, filling, T, w=None):
    import torch
    d = torch.from_numpy(np.ascontiguousarray(bands.T)).cuda()
    dw = None if w is None else torch.from_numpy(np.ascontiguousarray(w)).cuda()
    torch.cuda.synchronize()
    mu = ctypes.c_double()
    ctx.check(lqm.lib().lqm_chemicalpotential_bands_dev(ctx.handle, bands.shape[0], bands.shape[1], lqm._ptr(d),
                                                         lqm._ptr(dw), filling, T, ctypes.byref(mu)))
    return mu.value


# one value; one CTA and two; every CTA; the values of a CTA in and beyond shared memory
SHAPES = [(1, 1), (2, 3), (8, 128), (5, 205), (16, 9473), (31, 20011), (64, 9600)]


@pytest.mark.parametrize("n,nk", SHAPES)
def test_search_matches_oracle(lqm, ctx, n, nk):
    """T = 0: the same midpoint of order statistics, exactly.  T > 0: both are roots of the
    same filling to its rounding, so mu agrees to 1e-10 over a filling that rises."""
    rng = np.random.default_rng(n * nk)
    bands = np.sort(rng.normal(size=(n, nk)), axis=0)
    for filling in (0.0, 0.1, 0.5, 0.83, 1.0):
        # (a single value has no second order statistic in the oracle: it is its own neighbour)
        ref = bands[0, 0] if n * nk == 1 and 0 < filling < 1 else K.chemicalpotential(bands, filling, 0.0)
        assert device_mu(lqm, ctx, bands, filling, 0.0) == ref, filling
    if n * nk > 2:
        for filling in (0.2, 0.5, 0.77):
            mu, ref = device_mu(lqm, ctx, bands, filling, 0.05), K.chemicalpotential(bands, filling, 0.05)
            assert abs(mu - ref) <= 1e-10 * max(1.0, abs(ref)), filling
        w = rng.uniform(0.5, 1.5, nk)
        w /= w.sum()
        mu, ref = device_mu(lqm, ctx, bands, 0.4, 0.1, w), K.chemicalpotential(bands, 0.4, 0.1, w)
        assert abs(mu - ref) <= 1e-10 * max(1.0, abs(ref))


def test_search_with_ties(lqm, ctx):
    """Repeated values at T = 0: neighbouring order statistics that are equal, that differ,
    and all values the same."""
    bands = np.repeat(np.arange(-3.0, 3.0)[:, None], 500, axis=1)
    for filling in (0.1, 1 / 6, 0.4, 0.5, 0.66, 0.99):
        assert device_mu(lqm, ctx, bands, filling, 0.0) == K.chemicalpotential(bands, filling, 0.0), filling
    assert device_mu(lqm, ctx, np.full((3, 7), 0.25), 0.5, 0.0) == 0.25


def test_search_without_a_root_reports(lqm, ctx):
    """No sign change between the smallest and the largest value: the status of before."""
    bands = np.linspace(-1.0, 1.0, 64).reshape(4, 16)
    with pytest.raises(lqm.LQMError) as e:
        device_mu(lqm, ctx, bands, 1.5, 0.01)
    assert e.value.status == -6
