"""The autotuner's choice as a program saves it: another context given it runs the same kernels."""
import numpy as np
import pytest

from test_gpu_odd_orders import vacancy_cell

pytestmark = pytest.mark.gpu


def rho_of(lqm, c, h, ks):
    rho = {R: None for R in h}
    lqm.getdensitymatrix(rho, h, ks, mu=0.0, T=0.01, ctx=c)
    return rho


@pytest.mark.parametrize("n", [2, 24, 96, 150])
def test_saved_choice_replays_the_tuned_path(lqm, n):
    """Bit-identical rho; the reported choice is never slower than the best block size's
    kernel by construction, so an order left to the rule reports 0."""
    h = vacancy_cell(n, seed=n)
    rng = np.random.default_rng(n)
    tuned, fresh = lqm.Context(0, timeout=600), lqm.Context(0, timeout=600)
    best, ms, table = lqm.autotune_eigh(h, rng.uniform(-0.5, 0.5, (2, 600)), ctx=tuned)
    choice = tuned.eigh_threads(n)
    assert choice in (0, best) and ms == table[best]
    if n in (2, 150):  # the rule is the one-CTA kernel itself
        assert choice == best
    fresh.set_eigh_threads(n, choice)
    assert fresh.eigh_threads(n) == choice
    ks = rng.uniform(-0.5, 0.5, (2, 40))
    a, b = rho_of(lqm, tuned, h, ks), rho_of(lqm, fresh, h, ks)
    assert all(np.array_equal(a[R], b[R]) for R in h)
    tuned.reset_stats(timing=False)
    fresh.reset_stats(timing=False)
    rho_of(lqm, tuned, h, ks)
    rho_of(lqm, fresh, h, ks)
    assert tuned.stats()[1:] == fresh.stats()[1:]  # the same kernels
    tuned.close()
    fresh.close()


def test_fixed_reduction_below_224_tunes_block_sizes(lqm):
    """Accepted for every order that the one-CTA kernel takes, refused beyond."""
    c = lqm.Context(0, timeout=600)
    c.set_two_stage(1)
    h = vacancy_cell(170)
    best, _, table = lqm.autotune_eigh(h, np.random.default_rng(0).uniform(-0.5, 0.5, (2, 40)), ctx=c)
    assert best in table and best >= 32 and c.eigh_threads(170) in (0, best)
    with pytest.raises(lqm.LQMError):
        lqm.autotune_eigh(vacancy_cell(224), np.zeros((2, 1)), ctx=c)
    c.close()
