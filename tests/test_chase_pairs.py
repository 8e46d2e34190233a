"""The bulge chase's pairs of workers, as the device kernel runs them, on host threads."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emul(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pairs") / "libemul.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-I",
                    os.path.join(ROOT, "latticeqm.jl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "eigh_emul.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


def chase(emul, n, b, pairs, seed, limit=0):
    rng = np.random.default_rng(n + b)
    band = np.zeros((2 * b, n), complex, order="F")  # element (i, j) at [i - j, j]
    for o in range(min(b + 1, n)):
        band[o, : n - o] = rng.normal(size=n - o) + (1j * rng.normal(size=n - o) if o > 0 else 0.0)
    return emul.lqm_emul_chase_pairs(n, b, band.ctypes.data_as(ctypes.c_void_p), pairs, seed, ctypes.c_longlong(limit))


@pytest.mark.parametrize("b,n", [(4, 2), (4, 6), (4, 61), (16, 18), (16, 33), (16, 131), (16, 200)])
def test_pairs_match_the_sequential_chase(emul, b, n):
    """Band, reflectors and taus bit for bit, for the kernel's eight pairs and other counts."""
    for pairs, seed in ((8, 1), (8, 2), (1, 3), (2, 4), (3, 5), (13, 6)):
        assert chase(emul, n, b, pairs, seed) == 1, (pairs, seed)


def test_a_wait_that_expires_ends_every_pair(emul):
    """A limit of a few polls: whichever waits run out, all workers return (else the test hangs:
    an applier still on its way from the last meeting has to come to the maker's final one)."""
    ended = [chase(emul, 131, 16, 8, seed, limit=1 + seed % 3) for seed in range(600)]
    assert set(ended) <= {1, 2} and 2 in ended
