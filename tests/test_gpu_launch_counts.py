"""The launch counter against the kernels that each call launches."""
import numpy as np
import pytest

from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


def launches(c, call):
    c.reset_stats(timing=False)
    call()
    return c.stats()[2]


@pytest.mark.parametrize("n,one_cta", [(24, False), (96, False), (24, True)])
def test_every_kernel_is_counted_once(lqm, n, one_cta):
    c = lqm.Context(0, timeout=600)
    if one_cta:
        c.set_blocked_min_n(10 ** 9)
    h = vacancy_cell(n)
    H = lqm.DeviceHops(h, c)
    ks = np.random.default_rng(0).uniform(-0.5, 0.5, (2, 16))
    more = np.random.default_rng(0).uniform(-0.5, 0.5, (2, 1100))
    rho = {R: None for R in h}
    # reduction, divide and conquer, check of the leaves; factors, back-transformation; rho_k
    bands, vec, dens = (1, 1, 1) if one_cta else (3, 5, 6)
    assert launches(c, lambda: lqm.bandmatrix(H, ks, ctx=c)) == bands
    assert launches(c, lambda: lqm.bandmatrix(H, ks, want_vectors=True, ctx=c)) == vec
    # weights, band energy, fold coefficients, fold; its sum where k is split
    assert launches(c, lambda: lqm.getdensitymatrix(rho, H, ks, mu=0.0, T=0.01, ctx=c)) == dens + 4
    assert launches(c, lambda: lqm.getdensitymatrix(rho, H, more, mu=0.0, T=0.01, ctx=c)) == dens + 5
    assert launches(c, lambda: lqm.chemicalpotential(H, ks, 0.5, T=0.02, ctx=c)) == bands + 1
    H.free()
    c.close()
