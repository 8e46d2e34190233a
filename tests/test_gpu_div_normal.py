"""The branch-free quotient of the merges and the Lorentzian sums against IEEE division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P = ctypes.c_void_p


@pytest.fixture(scope="module")
def divlib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("div") / "libdiv.so")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "latticeqm.jl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "div_normal.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def test_builds(divlib):
    assert divlib.div_normal


def operands(kind, m, rng):
    sign = rng.choice([-1.0, 1.0], m)
    if kind == "poles":       # differences of scaled eigenvalues: both of any size down to 1e-150
        return sign * 10.0 ** rng.uniform(-150, 2, m), 10.0 ** rng.uniform(-150, 2, m)
    if kind == "wide":        # x^2 + width^2 up to the largest that the Lorentzian sums admit
        return sign * 10.0 ** rng.uniform(-5, 150, m), 10.0 ** rng.uniform(-150, 300, m)
    if kind == "narrow":      # and down to the smallest
        return sign * 10.0 ** rng.uniform(-145, -5, m), 10.0 ** rng.uniform(-290, -150, m)
    if kind == "near one":    # quotients around a power of two, where the spacing changes
        a = 1.0 + rng.integers(0, 2**12, m) * 2.0**-52
        return sign * a, 1.0 + rng.integers(0, 2**12, m) * 2.0**-52
    return rng.integers(1, 2**53, m).astype(float), sign * rng.integers(1, 2**53, m).astype(float)  # full mantissas


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["poles", "wide", "narrow", "near one", "mantissas"])
def test_quotient_within_one_place(divlib, kind):
    """The corrected quotient is within half a place and 2^-49 of one of the exact value
    (Newton's reciprocal to 2 places, its quotient to 4, times the residual's error): at most
    one place off IEEE's, and off at all only next to a tie, less than once in a million."""
    m = 1 << 22
    a, b = operands(kind, m, np.random.default_rng(7))
    q = np.empty(m)
    assert divlib.div_normal(a.ctypes.data_as(P), b.ctypes.data_as(P), q.ctypes.data_as(P), ctypes.c_longlong(m)) == 0
    ref = a / b
    assert np.all(np.abs(ref) >= np.finfo(float).tiny)
    off = q.view(np.int64) - ref.view(np.int64)
    assert np.max(np.abs(off)) <= 1 and np.count_nonzero(off) <= m // 1000000
