"""Divide and conquer on a tridiagonal with NaN or infinite entries: every index that a later
step or kernel reads has to stay in range (the values are lost, the memory is not)."""
import ctypes

import numpy as np
import pytest

from test_emulation import emul  # noqa: F401

P = ctypes.c_void_p


def solve(lib, d, e, tile_min):
    n = len(d)
    idx, ev, Z = np.zeros((5, n), np.int32), np.zeros(n), np.zeros((n, n), order="F")
    bad = lib.lqm_emul_dc_root(n, d.ctypes.data_as(P), e.ctypes.data_as(P), tile_min, idx.ctypes.data_as(P),
                               ev.ctypes.data_as(P), Z.ctypes.data_as(P))
    return bad, idx, ev, Z


def entries(n, where):
    rng = np.random.default_rng(n)
    d, e = rng.normal(size=n), rng.normal(size=n - 1)
    if where == "all":
        d[:], e[:] = np.nan, np.nan
    elif where == "tail":  # what a reduction leaves of one NaN element
        d[1:], e[1:] = np.nan, np.nan
    elif where == "d":
        d[n // 3] = np.nan
    elif where == "e":
        e[(n - 1) // 2] = np.nan
    elif where == "-nan":
        d[:] = np.copysign(np.nan, -1.0)
    elif where == "inf":
        d[0], d[n - 1], e[(n - 1) // 3] = np.inf, -np.inf, np.inf
    return d, e


@pytest.mark.parametrize("where", ["finite", "all", "tail", "d", "e", "-nan", "inf"])
@pytest.mark.parametrize("n", [2, 7, 33, 64, 161])
def test_merge_indices_stay_in_range(emul, n, where):  # noqa: F811
    d, e = entries(n, where)
    bad, idx, ev, Z = solve(emul, d, e, 1)
    assert bad == 0
    assert sorted(idx[2]) == list(range(n))      # the last merge's places are a permutation
    assert np.all((idx[0] >= 0) & (idx[0] < n))  # and no hole is left in its merged order
    if where == "finite":
        A = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
        assert np.max(np.abs(ev - np.linalg.eigvalsh(A))) <= 1e-13 * max(1.0, n)
        assert np.max(np.abs(A @ Z - Z * ev)) <= 1e-13 * max(1.0, n)
