"""The staged eigensolver (n <= 144) at the edges of its thread grids, leaves and tiles."""
import numpy as np
import pytest

from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu
BAND_TOL = 1e-10  # of the spectral width, as in test_gpu_parity
RHO_TOL = 1e-9

# one past and at: a warp's row blocks (8 .. 32), a CTA's (48 .. 144), leaves of 16 and 17,
# the divide-and-conquer CTA sizes (32, 64, 96), the back-transformation's row tiles
ORDERS = [3, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 113, 128, 129, 144]


@pytest.mark.parametrize("n", ORDERS)
def test_staged_path_matches_oracle(lqm, ctx, n):
    """Eigenpairs, eigenvalues alone, and rho with nearly all, nearly no, all and no states
    full (its direct and complement forms and their empty cases)."""
    h = vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, 5))
    b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=ctx)
    ref, _ = K.bandmatrix(h, ks)
    width = np.ptp(ref)
    assert np.max(np.abs(b - ref)) <= BAND_TOL * width
    assert np.max(np.abs(lqm.bandmatrix(h, ks, ctx=ctx)[0] - ref)) <= BAND_TOL * width
    for j in range(ks.shape[1]):
        Hk = K.fouriersum(h, ks[:, j])
        assert np.max(np.abs(Hk @ U[:, :, j] - U[:, :, j] * b[:, j])) <= BAND_TOL * width
        assert np.max(np.abs(U[:, :, j].conj().T @ U[:, :, j] - np.eye(n))) <= 1e-12
    w = np.full(5, 0.2)
    for mu, T in ((0.0, 0.01), (0.4 * ref.max(), 0.02), (0.4 * ref.min(), 0.02), (2 * ref.max(), 0.01),
                  (2 * ref.min() - 1, 0.01), (0.1, 0.0)):
        rho = {R: None for R in h}
        e = lqm.getdensitymatrix(rho, h, ks, mu=mu, T=T, ctx=ctx)
        rref, eref = K.densitymatrix(h, ks, w, mu, T, list(h.keys()))
        assert max(np.max(np.abs(rho[R] - rref[R])) for R in h) <= RHO_TOL
        assert abs(e - eref) <= 1e-9 * max(1.0, n * width)
