"""Eigen passes beside a program that holds nearly all of the device's memory: the passes'
batches shrink to what is left instead of the call being refused."""
import numpy as np
import pytest

from lqm_workloads import lattice as L
from oracle import kspace as K
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nk", [(96, 128 * 128), (176, 128 * 128)])
@pytest.mark.parametrize("vectors", [False, True])
def test_passes_fit_the_memory_that_is_left(lqm, n, nk, vectors):
    """1.5 GB left, below one full batch of either path (2.5 to 5 and 20 to 40 GB here): bands,
    or rho_L and with it the eigenvectors, equal the oracle on every 1000th k-point and the
    unconstrained call to rounding."""
    import torch
    h = vacancy_cell(n, seed=n)
    ks = L.regulargrid(nk)
    ref, _ = K.bandmatrix(h, ks[:, ::1000])
    width = np.ptp(ref)

    def call(c):
        if not vectors:
            return lqm.bandmatrix(h, ks, ctx=c)[0], None
        rho = {(0, 0): None}
        lqm.getdensitymatrix(rho, h, ks, mu=0.0, T=0.05, ctx=c)
        return None, rho[(0, 0)]

    free = lqm.Context(0, timeout=600)
    b0, r0 = call(free)
    free.close()
    torch.cuda.empty_cache()
    c = lqm.Context(0, timeout=600)
    held = []
    try:
        left = (1.5 + (4.5 if vectors else 0.0)) * 2**30  # rho_k of a batch is up to 4 GB by itself
        while torch.cuda.mem_get_info()[0] > left + 2**28:
            held.append(torch.empty(int(min(torch.cuda.mem_get_info()[0] - left, 2**33)), dtype=torch.uint8,
                                    device="cuda"))
        b, r = call(c)
    finally:
        held.clear()
        torch.cuda.empty_cache()
        c.close()
    if vectors:
        assert np.max(np.abs(r - r0)) <= 1e-12
    else:
        assert np.max(np.abs(b - b0)) <= 1e-12 * width
        assert np.max(np.abs(b[:, ::1000] - ref)) <= 1e-10 * width


def test_a_refused_call_is_not_reported_again(lqm):
    """Eigenvectors of 2.4 GB with 0.5 GB left are refused; the next call, on the same and on
    another context, is served."""
    import torch
    h = vacancy_cell(96)
    c = lqm.Context(0, timeout=600)
    small = L.regulargrid(4)
    want = lqm.bandmatrix(h, small, ctx=c)[0]
    held = []
    try:
        torch.cuda.empty_cache()
        while torch.cuda.mem_get_info()[0] > 2**29 + 2**28:
            held.append(torch.empty(int(min(torch.cuda.mem_get_info()[0] - 2**29, 2**33)), dtype=torch.uint8,
                                    device="cuda"))
        with pytest.raises(lqm.LQMError, match="ENOMEM"):
            lqm.bandmatrix(h, L.regulargrid(128 * 128), want_vectors=True, ctx=c)
        assert np.array_equal(lqm.bandmatrix(h, small, ctx=c)[0], want)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    other = lqm.Context(0, timeout=600)
    assert np.array_equal(lqm.bandmatrix(h, small, ctx=other)[0], want)
    other.close()
    c.close()
