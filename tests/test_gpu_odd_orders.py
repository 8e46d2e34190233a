"""Passes with eigenvectors at odd orders on the one-CTA eigensolver (its per-CTA scratch
slots hold 16-byte elements, so their stride has to be a whole number of them)."""
import numpy as np
import pytest

from lqm_workloads import lattice as L
from lqm_workloads import models as M
from oracle import kspace as K

pytestmark = pytest.mark.gpu


def vacancy_cell(n, seed=0):
    """A honeycomb cell cut to n orbitals, with on-site disorder."""
    side = 1
    while 2 * side * side < n:
        side += 1
    lat = L.superlattice(L.honeycomb(), [side, side])
    h = M.graphene(lat, tz=0.0, tmin=1e-3)
    rng = np.random.default_rng(seed)
    keep = np.sort(rng.permutation(lat.norb)[:n])
    h = {R: B[np.ix_(keep, keep)] for R, B in h.items()}
    h[(0, 0)] = h[(0, 0)] + np.diag(rng.normal(0.0, 0.1, n))
    return h


@pytest.mark.parametrize("n", [3, 5, 25, 51])
def test_one_cta_kernel_at_odd_orders(lqm, n):
    """Eigenpairs of several k-points per CTA wave: residual 1e-10 of the spectral width."""
    c = lqm.Context(0, timeout=600)
    try:
        c.set_blocked_min_n(10 ** 9)  # the one-CTA kernel
        h = vacancy_cell(n)
        ks = np.random.default_rng(1).uniform(-0.5, 0.5, (2, 40))
        b, U = lqm.bandmatrix(h, ks, want_vectors=True, ctx=c)
        ref, _ = K.bandmatrix(h, ks)
        width = np.ptp(ref)
        assert np.max(np.abs(b - ref)) <= 1e-10 * width
        for j in range(ks.shape[1]):
            Hk = K.fouriersum(h, ks[:, j])
            assert np.max(np.abs(Hk @ U[:, :, j] - U[:, :, j] * b[:, j])) <= 1e-10 * width
    finally:
        c.close()
