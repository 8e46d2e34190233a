"""NaN in a k-list, or an overflow in H(k): the k-point's own results are lost, nothing else is."""
import numpy as np
import pytest

from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu

# the staged path's warp, CTA and 16-warp forms; the one-CTA kernel with its matrix in shared
# and in global memory; the blocked path with plain and with tiled merges
CASES = [(9, None), (24, None), (40, None), (96, None), (144, None), (40, "one"), (150, "one"), (40, "blocked"),
         (200, "blocked")]


def context(lqm, path):
    c = lqm.Context(0, timeout=600)
    if path:
        c.set_blocked_min_n(1 if path == "blocked" else 10 ** 9)
    return c


def solve(lqm, c, H, n, ks):
    import torch
    nk = ks.shape[1]
    d_ks = torch.from_numpy(np.ascontiguousarray(ks.T)).cuda()
    b = torch.zeros(nk, n, dtype=torch.float64, device="cuda")
    U = torch.zeros(nk, n, n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    c.check(lqm.lib().lqm_bandmatrix_dev(c.handle, H.handle, nk, lqm._ptr(d_ks), 1, 0, lqm._ptr(b), lqm._ptr(U)))
    torch.cuda.synchronize()
    return b.cpu().numpy(), U.cpu().numpy()


@pytest.mark.parametrize("n,path", CASES)
def test_nan_k_points_leave_the_others(lqm, n, path):
    """Bands and eigenvectors of the finite k-points are those of a list without NaN, bit for bit."""
    c = context(lqm, path)
    H = lqm.DeviceHops(vacancy_cell(n, seed=n), c)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, 7))
    bad = ks.copy()
    bad[0, 0] = bad[1, 3] = bad[0, 6] = np.nan
    b0, U0 = solve(lqm, c, H, n, ks)
    b1, U1 = solve(lqm, c, H, n, bad)
    ok = [1, 2, 4, 5]
    assert np.array_equal(b0[ok], b1[ok]) and np.array_equal(U0[ok], U1[ok])
    H.free()
    c.close()


@pytest.mark.parametrize("n,path", CASES)
def test_overflow_then_a_finite_matrix(lqm, n, path):
    """One on-site energy whose Bloch sum overflows (part of the tridiagonal stays finite), with
    occupations that split the finite part; the context then gives the oracle's rho of a
    finite matrix."""
    c = context(lqm, path)
    h = vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, 5))
    for site in (0, n // 2, n - 1):
        broken = {R: B.copy() for R, B in h.items()}
        for R in ((0, 0), (1, 0), (-1, 0)):
            broken[R][site, site] = 1.7e308
        for mu in (-100.0, 0.0, 100.0):
            lqm.getdensitymatrix({R: None for R in h}, broken, np.zeros((2, 3)), mu=mu, T=0.01, ctx=c)
    rho = {R: None for R in h}
    lqm.getdensitymatrix(rho, h, ks, mu=0.0, T=0.01, ctx=c)
    rref, _ = K.densitymatrix(h, ks, np.full(5, 0.2), 0.0, 0.01, list(h.keys()))
    assert max(np.max(np.abs(rho[R] - rref[R])) for R in h) <= 1e-9
    c.close()
