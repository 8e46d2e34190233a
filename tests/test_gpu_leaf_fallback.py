"""The staged path's fallback: k-points of which a leaf's QL iteration did not end are solved
again by the one-CTA kernel, here by a limit on the sweeps."""
import numpy as np
import pytest

from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell
from test_gpu_staged import BAND_TOL, RHO_TOL

pytestmark = pytest.mark.gpu


def two_chains(n):
    """Diagonal at k = 0 (no sweep is needed there), coupled everywhere else."""
    d = np.linspace(-1.0, 1.0, n)
    A = 0.3 * np.eye(n, k=1)
    return {(0, 0): np.diag(d) + 0j, (1, 0): A + 0j, (-1, 0): A.T + 0j, (0, 1): -(A + A.T) / 2 + 0j,
            (0, -1): -(A + A.T) / 2 + 0j}


@pytest.mark.parametrize("n", [3, 16, 17, 40, 72, 96, 144])
@pytest.mark.parametrize("mixed", [False, True])
def test_redone_points_match_oracle(lqm, n, mixed):
    """One sweep per leaf: every k-point (or, mixed, all but those at k = 0) is redone.
    Bands, eigenvectors, rho in its direct, complement and all-vectors forms, band energy."""
    h = two_chains(n) if mixed else vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(0.1, 0.4, (2, 7))
    if mixed:
        ks[:, [0, 3]] = 0.0
    c, plain = lqm.Context(0, timeout=600), lqm.Context(0, timeout=600)
    c.set_leaf_sweeps(1)
    ref, _ = K.bandmatrix(h, ks)
    width = np.ptp(ref)
    b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=c)
    assert np.max(np.abs(b - ref)) <= BAND_TOL * width
    assert np.max(np.abs(lqm.bandmatrix(h, ks, ctx=c)[0] - ref)) <= BAND_TOL * width
    for j in range(ks.shape[1]):
        Hk = K.fouriersum(h, ks[:, j])
        assert np.max(np.abs(Hk @ U[:, :, j] - U[:, :, j] * b[:, j])) <= BAND_TOL * width
        assert np.max(np.abs(U[:, :, j].conj().T @ U[:, :, j] - np.eye(n))) <= 1e-12
    w = np.full(7, 1.0 / 7)
    for mu, T in ((0.4 * ref.min(), 0.02), (0.4 * ref.max(), 0.02), (0.1, 0.0)):
        rho = {R: None for R in h}
        e = lqm.getdensitymatrix(rho, h, ks, mu=mu, T=T, ctx=c)
        rref, eref = K.densitymatrix(h, ks, w, mu, T, list(h.keys()))
        assert max(np.max(np.abs(rho[R] - rref[R])) for R in h) <= RHO_TOL
        assert abs(e - eref) <= 1e-9 * max(1.0, n * width)
    # the points that need no sweep are the staged path's, bit for bit
    if mixed:
        b0, U0 = lqm.bandmatrix(h, ks, want_vectors=True, ctx=plain)
        assert np.array_equal(b[:, [0, 3]], b0[:, [0, 3]]) and np.array_equal(U[:, :, [0, 3]], U0[:, :, [0, 3]])
    # the limit taken back: the staged results again
    c.set_leaf_sweeps(0)
    assert np.array_equal(lqm.bandmatrix(h, ks, ctx=c)[0], lqm.bandmatrix(h, ks, ctx=plain)[0])
    c.close()
    plain.close()
