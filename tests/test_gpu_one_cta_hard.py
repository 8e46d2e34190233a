"""The hard Hermitian inputs of the emulation suite on the one-CTA eigensolver, which orders
up to 144 reach where a block size is set (or, beyond 512 keys, by default)."""
import numpy as np
import pytest

from oracle import kspace as K
from test_emulation import _hard_hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [32, 128, 512])
def test_hard_hermitian_inputs_on_the_one_cta_kernel(lqm, nt):
    c = lqm.Context(0, timeout=600)
    for name, Hk in _hard_hermitian():
        n = Hk.shape[0]
        c.set_eigh_threads(n, nt)
        c.reset_stats(timing=False)
        b, U = lqm.bandmatrix({(0, 0): Hk}, np.zeros((2, 1)), want_vectors=True, ctx=c)
        assert c.stats()[2] == 1, name  # one kernel: not the staged path
        ref = K.eigh_upper(Hk, vectors=False)
        scale = max(np.max(np.abs(ref)), np.finfo(float).tiny)
        Uk = U[:, :, 0]
        assert np.max(np.abs(b[:, 0] - ref)) <= 1e-12 * scale, name
        assert np.max(np.abs(Uk.conj().T @ Uk - np.eye(n))) <= 1e-12, name
        assert np.max(np.abs(Hk @ Uk - Uk * b[:, 0])) <= 1e-12 * scale, name
    c.close()
