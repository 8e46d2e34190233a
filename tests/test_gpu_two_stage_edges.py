"""The two-stage eigensolver at the edges of its panels, their blocks and the column blocks
of its back-transformation."""
import numpy as np
import pytest

from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu
BAND_TOL = 1e-10  # of the spectral width, as in test_gpu_parity
RHO_TOL = 1e-9

# bands of 16: one row below the first panel (18), short last panels (31 .. 49); column
# blocks of 128 (144, 145); panels of 512 rows in one block and of 513 and more in
# two (528, 529), of 1025 in three (1041); the last merge in a kernel of its own from 160 on,
# its row tiles of 128 per child and column tiles of 64 (160, 161, 256, 257, 385)
ORDERS = [18, 31, 32, 33, 48, 49, 144, 145, 160, 161, 256, 257, 385, 528, 529, 1041]


@pytest.mark.parametrize("n", ORDERS)
def test_two_stage_matches_oracle(lqm, n):
    c = lqm.Context()
    c.set_blocked_min_n(1)
    c.set_two_stage(1)
    nk = 3 if n < 500 else 2
    h = vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, nk))
    b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=c)
    ref, _ = K.bandmatrix(h, ks)
    width = np.ptp(ref)
    assert np.max(np.abs(b - ref)) <= BAND_TOL * width
    assert np.max(np.abs(lqm.bandmatrix(h, ks, ctx=c)[0] - ref)) <= BAND_TOL * width
    for j in range(nk):
        Hk = K.fouriersum(h, ks[:, j])
        assert np.max(np.abs(Hk @ U[:, :, j] - U[:, :, j] * b[:, j])) <= BAND_TOL * width
        assert np.max(np.abs(U[:, :, j].conj().T @ U[:, :, j] - np.eye(n))) <= 1e-12 * max(1.0, n / 144)
    w = np.full(nk, 1.0 / nk)
    for mu in (0.0, 0.4 * ref.max()):  # half and nearly all states full
        rho = {R: None for R in h}
        e = lqm.getdensitymatrix(rho, h, ks, mu=mu, T=0.01, ctx=c)
        rref, eref = K.densitymatrix(h, ks, w, mu, 0.01, list(h.keys()))
        assert max(np.max(np.abs(rho[R] - rref[R])) for R in h) <= RHO_TOL
        assert abs(e - eref) <= 1e-9 * max(1.0, n * width)
    c.close()


@pytest.mark.parametrize("levels", [1, 2, 7, 150])
def test_merges_with_degenerate_levels(lqm, levels):
    """A 300 x 300 matrix with `levels` distinct eigenvalues: merges that deflate nearly
    everything or everything, with rotations between columns of both children."""
    n = 300
    rng = np.random.default_rng(levels)
    q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    d = np.sort(np.linspace(-1.0, 1.0, levels)[rng.integers(0, levels, n)])
    H = (q * d) @ q.conj().T
    h = {(0, 0): 0.5 * (H + H.conj().T)}
    ks = np.zeros((2, 2))
    for mode in (1, 0):
        c = lqm.Context()
        c.set_blocked_min_n(1)
        c.set_two_stage(mode)
        b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=c)
        assert np.max(np.abs(b[:, 0] - d)) <= 1e-12
        for j in range(2):
            assert np.max(np.abs(h[(0, 0)] @ U[:, :, j] - U[:, :, j] * b[:, j])) <= 1e-12
            assert np.max(np.abs(U[:, :, j].conj().T @ U[:, :, j] - np.eye(n))) <= 2e-12
        c.close()


@pytest.mark.parametrize("n", [159, 160, 223])
def test_orders_at_the_default_switch(lqm, n):
    """The one-CTA kernel, the blocked path, and the one-CTA kernel kept by a set block size."""
    h = vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, 3))
    ref, _ = K.bandmatrix(h, ks)
    width = np.ptp(ref)
    rref, eref = K.densitymatrix(h, ks, np.full(3, 1 / 3), 0.1, 0.01, list(h.keys()))
    for threads in (0, 384):
        c = lqm.Context()
        if threads:
            c.set_eigh_threads(n, threads)
        b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=c)
        assert np.max(np.abs(b - ref)) <= BAND_TOL * width
        assert np.max(np.abs(lqm.bandmatrix(h, ks, ctx=c)[0] - ref)) <= BAND_TOL * width
        for j in range(3):
            Hk = K.fouriersum(h, ks[:, j])
            assert np.max(np.abs(Hk @ U[:, :, j] - U[:, :, j] * b[:, j])) <= BAND_TOL * width
        rho = {R: None for R in h}
        e = lqm.getdensitymatrix(rho, h, ks, mu=0.1, T=0.01, ctx=c)
        assert max(np.max(np.abs(rho[R] - rref[R])) for R in h) <= RHO_TOL
        assert abs(e - eref) <= 1e-9 * max(1.0, n * width)
        c.close()
