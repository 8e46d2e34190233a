"""Batched products of the library's GEMM at orders on each of its tile shapes and remainders."""
import numpy as np
import pytest

from lqm_workloads import lattice as L
from oracle import kspace as K
from oracle import meanfield as MF
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [66, 72, 73, 96, 97, 100, 144, 145, 200, 216, 264, 400])
def test_commutator_norm_matches_oracle(lqm, ctx, n):
    """Two products per k-point, 1e-12 relative (sums of n terms, rounding 1e-16 sqrt(n) each)."""
    h = vacancy_cell(n, seed=n)
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    rho = {(0, 0): a + a.conj().T}
    ks = L.regulargrid(9)
    ref = MF.commutator_kspace_norm(h, rho, ks)
    assert abs(lqm.commutator_kspace_norm(h, rho, ks, ctx=ctx) - ref) <= 1e-12 * ref


@pytest.mark.parametrize("n,nk,nkeys", [(180, 9, 5), (182, 9, 5), (182, 64, 16), (182, 260, 3), (190, 16, 33), (190, 70, 35)])
def test_fold_on_tall_tiles_matches_oracle(lqm, ctx, n, nk, nkeys):
    """rho_L at orders around 181 (n^2 = 32768 rows), short and longer k, few and many keys."""
    h = vacancy_cell(n, seed=n)
    ks = np.random.default_rng(n).uniform(-0.5, 0.5, (2, nk))
    keys = [(i, j) for i in range(-3, 4) for j in range(-3, 4)][:nkeys]
    rho = {R: None for R in keys}
    e = lqm.getdensitymatrix(rho, h, ks, mu=0.0, T=0.05, ctx=ctx)
    ref, eref = K.densitymatrix(h, ks, np.full(nk, 1.0 / nk), 0.0, 0.05, keys)
    assert max(np.max(np.abs(rho[R] - ref[R])) for R in keys) <= 1e-9
    assert abs(e - eref) <= 1e-9 * max(1.0, abs(eref))
