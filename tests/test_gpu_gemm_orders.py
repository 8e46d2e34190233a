"""Batched products of the library's GEMM at orders on each of its tile shapes and remainders."""
import numpy as np
import pytest

from lqm_workloads import lattice as L
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
