"""The several-models call (lqm_bands_dos_rho_multi_dev) on each kernel it can take."""
import numpy as np
import pytest

from oracle import kspace as K
from lqm_workloads import lattice as L
from test_gpu_multi import GAMMA, MU, TEMP, _state
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


def run(lqm, c, models, ks):
    import torch
    dev = torch.device("cuda", 0)
    d_ks = torch.from_numpy(np.ascontiguousarray(ks.T)).to(dev)
    st = [_state(lqm, c, torch, dev, h, ks.shape[1]) for h in models]
    eb = lqm.bands_dos_rho_multi_dev(st, d_ks, ks.shape[1], mu=MU, T=TEMP, gamma=GAMMA, ctx=c)
    return st, eb, d_ks


def check(st, eb, ks):
    nk = ks.shape[1]
    for s, e in zip(st, eb):
        b_ref, _ = K.bandmatrix(s["h"], ks)
        assert np.max(np.abs(s["bands"].cpu().numpy().T - b_ref)) <= 1e-10 * np.ptp(b_ref), s["n"]
        keys = list(s["h"].keys())
        rref, ebref = K.densitymatrix(s["h"], ks, np.full(nk, 1.0 / nk), MU, TEMP, keys)
        got = s["rho"].cpu().numpy()
        assert max(np.max(np.abs(got[i].T - rref[R])) for i, R in enumerate(keys)) <= 1e-9, s["n"]
        assert abs(e - ebref) <= 1e-9 * max(1.0, abs(ebref)), s["n"]


@pytest.mark.parametrize("orders", [(160,), (24, 176), (2, 96, 150), (223, 8)])
def test_orders_up_to_223_are_served(lqm, ctx, orders):
    ks = L.regulargrid(9)
    st, eb, _ = run(lqm, ctx, [vacancy_cell(n, seed=n) for n in orders], ks)
    check(st, eb, ks)


def test_orders_from_224_on_are_refused(lqm, ctx):
    for orders, n_min in (((224,), 0), ((24, 224), 0), ((24, 40), 40)):
        c = lqm.Context(0, timeout=600)
        c.set_blocked_min_n(n_min)
        with pytest.raises(lqm.LQMError) as e:
            run(lqm, c, [vacancy_cell(n, seed=n) for n in orders], L.regulargrid(4))
        assert e.value.status == -1
        c.close()
