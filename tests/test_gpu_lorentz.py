"""Lorentzian sums (DOS, conductivity): the widths, frequencies and energies at which the
kernels leave their branch-free quotients, and the pairs of equal occupation they skip."""
import numpy as np
import pytest

import lqm_cuda as Q
from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [1e-160, 1e-146, 1e-3, 0.3, 1e149, 1e151])
def test_dos_of_given_bands(lqm, ctx, gamma):
    """1e-13 of the sum of the terms' magnitudes: a rounding or two per term, and their sum."""
    import torch
    rng = np.random.default_rng(3)
    n, nk, nw = 7, 301, 70
    bands = rng.normal(size=(nk, n))
    bands[0, 0], bands[200, 3], bands[250, 1] = np.inf, -np.inf, 1e170
    w = rng.uniform(0.5, 1.5, nk)
    om = np.concatenate([rng.normal(size=nw - 2), [1e151, -1e155]])
    db, dw, do = (torch.tensor(x, device="cuda") for x in (bands, w, om))
    out = torch.zeros(nw, device="cuda", dtype=torch.float64)
    ctx.check(Q._lib.lqm_dos_bands_dev(ctx.handle, n, nk, db.data_ptr(), dw.data_ptr(), nw, do.data_ptr(), gamma,
                                       out.data_ptr()))
    torch.cuda.synchronize()
    with np.errstate(over="ignore"):
        x = om[:, None, None] - bands[None]
        terms = w[None, :, None] * gamma / (x * x + gamma * gamma)
    ref = terms.sum((1, 2))
    scale = out.cpu().numpy()[0] / ref[0]  # the function's normalisation
    assert np.max(np.abs(out.cpu().numpy() / scale - ref) / np.maximum(np.abs(ref), 1e-290)) <= 1e-13


@pytest.mark.parametrize("T,mu", [(0.0, 0.1), (0.01, 0.0), (5.0, 0.0), (0.01, 50.0)])
def test_conductivity_with_empty_and_full_states(lqm, ctx, T, mu):
    """All, some, nearly no and only pairs of equal occupation: 1e-9 of the largest value."""
    n = 26
    h = vacancy_cell(n, seed=1)
    rng = np.random.default_rng(0)
    j1 = {R: 1j * rng.normal(size=(n, n)) for R in h}
    J = {R: j1[R] + np.conj(j1[tuple(-x for x in R)]).T for R in h}
    ks = rng.uniform(-0.5, 0.5, (2, 4))
    om = np.linspace(0.0, 2.0, 11)
    got = lqm.opticalconductivity(om, h, J, J, ks, mu=mu, Gamma=0.05, T=T, ctx=ctx)
    ref = K.opticalconductivity(om, h, J, J, ks, mu=mu, gamma=0.05, T=T)
    assert np.max(np.abs(got - ref)) <= 1e-9 * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("gamma", [1e-160, 1e-146, 0.05, 1e149, 1e151])
@pytest.mark.parametrize("top", [2.0, 1e149, 1e153, 1e170])
@pytest.mark.parametrize("far", [False, True])
def test_conductivity_of_distant_levels(lqm, ctx, gamma, top, far):
    """Uncoupled levels up to 1e170 (squares beyond the largest number: zero terms), widths and
    frequencies on both sides of the fast form's range: 1e-12 of the terms' magnitudes."""
    e = np.array([-top, -1.0, 0.3, 1.0, top])
    n = len(e)
    rng = np.random.default_rng(0)
    J = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    J = J + J.conj().T
    om = np.array([0.0, 0.61, 1e120, 1e151, -1e155][:5 if far else 3])  # one far frequency turns its whole tile
    got = lqm.opticalconductivity(om, {(0, 0): np.diag(e).astype(complex)}, {(0, 0): J}, {(0, 0): J}, np.zeros((2, 1)),
                                  mu=0.0, Gamma=gamma, T=0.0, ctx=ctx)
    f = (e < 0.0).astype(float)
    off = ~np.eye(n, dtype=bool)
    wt = ((f[:, None] - f[None, :]) * np.abs(J) ** 2)[off]
    with np.errstate(over="ignore"):
        z = (e[:, None] - e[None, :])[off][None] - om[:, None]
        r = 1.0 / (z * z + gamma * gamma)
        ref = -1j * (wt * (z + 1j * gamma) * r).sum(1)
        scale = (np.abs(wt) * (np.abs(z) + gamma) * r).sum(1)
    assert np.all(np.isfinite(got)) and np.all(np.abs(got - ref) <= 1e-12 * scale)
