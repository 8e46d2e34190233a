"""Host threads with a context each and different orders on the same kernels."""
import threading

import numpy as np
import pytest

from lqm_workloads import lattice as L
from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orders,nt", [((50, 64), 0), ((81, 96), 0), ((97, 144), 0), ((40, 72), 64)])
def test_orders_of_one_kernel_in_two_threads(lqm, orders, nt):
    """The limit of a kernel's dynamic shared memory is the process's, not the context's: no
    launch is refused, and every result is the one of the thread alone, bit for bit."""
    ks = L.regulargrid(16)
    hs = [vacancy_cell(n, seed=n) for n in orders]
    bad = []

    def one(c, h):
        rho = {R: None for R in h}
        lqm.getdensitymatrix(rho, h, ks, mu=0.0, T=0.02, ctx=c)
        return rho

    def work(h, n, expect, start):
        try:
            c = lqm.Context(0, timeout=60)
            c.set_eigh_threads(n, nt)
            start.wait(60)
            for _ in range(150):
                rho = one(c, h)
                if not all(np.array_equal(rho[R], expect[R]) for R in h):
                    bad.append((n, "another result"))
                    break
            c.close()
        except Exception as e:  # noqa: BLE001 - reported below
            bad.append((n, repr(e)))

    expect = []
    for h, n in zip(hs, orders):
        c = lqm.Context(0, timeout=60)
        c.set_eigh_threads(n, nt)
        expect.append(one(c, h))
        c.close()
    start = threading.Barrier(4)
    ts = [threading.Thread(target=work, args=(hs[i % 2], orders[i % 2], expect[i % 2], start)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(180)
    assert not bad, bad[:3]


def test_limit_is_raised_once_and_stays(lqm):
    """A small order after a large one on the same kernel, then the large one again."""
    ks = L.regulargrid(9)
    c = lqm.Context(0, timeout=60)
    first = {}
    for n in (96, 81, 96, 81):
        h = vacancy_cell(n, seed=n)
        b = lqm.bandmatrix(h, ks, ctx=c)[0]
        assert np.array_equal(first.setdefault(n, b), b)
    c.close()
