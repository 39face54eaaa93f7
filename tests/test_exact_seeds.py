"""The exact quotients and roots from every seed their proofs admit, on the
host: relative errors of either sign up to 2^-19 (kt_exact.cuh takes the
hardware's, checked on the device by test_gpu_exact_device.py)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import test_exact as te
import testlibs

SRC = os.path.join(testlibs.TESTS, "kt_seedcheck.cpp")
LIB = os.path.join(testlibs.BUILD, "libkt_seedcheck.so")
# the band's ends, a seed that is the correctly rounded value, and between
RELS = [s * 2.0 ** -19 * f for s in (-1, 1) for f in (1.0, 0.75, 0.5, 0.25, 2.0 ** -10)] + [0.0]


@pytest.fixture(scope="module")
def sc():
    os.makedirs(testlibs.BUILD, exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off", "-march=x86-64-v3",
                    "-shared", "-o", LIB, SRC], check=True)
    L = ctypes.CDLL(LIB)
    P, D, N = ctypes.c_void_p, ctypes.c_double, ctypes.c_long
    L.sc_quot.argtypes, L.sc_quot.restype = [N, P, P, D], N
    L.sc_sqrt.argtypes, L.sc_sqrt.restype = [N, P, D, ctypes.POINTER(D)], N
    return L


def quot_operands(n=200_000):
    """Denominators over the whole range and next to 1 and to the refused
    ones, numerators whose quotients lie next to a rounding midpoint."""
    rng = np.random.default_rng(12)
    b, a = te._bits(rng, n, -300, 300), te._bits(rng, n, -400, 400)
    b[: n // 8] = 2.0 - 2.0 ** -18 - np.arange(n // 8) * 2.0 ** -52
    b[n // 8: n // 4] = 1.0 + np.arange(n // 8) * 2.0 ** -52
    mid = np.ldexp(rng.integers(1 << 53, 1 << 54, n // 2).astype(np.float64), -53)
    a[: n // 2] = mid * b[: n // 2]
    a[-100:] = 0.0
    return a, b


def root_operands(n=100_000):
    rng = np.random.default_rng(13)
    hard = te._hard_roots()
    g = np.ldexp(rng.integers(1 << 53, 1 << 54, n).astype(np.float64), -53)
    # up to the refused ones below a power of four
    top = 4.0 - 2.0 ** -17 - np.arange(n) * 2.0 ** -51
    return np.ascontiguousarray(np.concatenate([hard, hard * 4.0, g * g, top, np.abs(te._bits(rng, n, -250, 250))]))


@pytest.mark.parametrize("rel", RELS)
def test_quotients_from_any_seed(sc, rel):
    a, b = quot_operands()
    assert sc.sc_quot(len(a), te._p(a), te._p(b), rel) == 0


@pytest.mark.parametrize("rel", RELS)
def test_roots_from_any_seed(sc, rel):
    x = root_operands()
    worst = ctypes.c_double()
    assert sc.sc_sqrt(len(x), te._p(x), rel, ctypes.byref(worst)) == 0
    assert worst.value < 1.41  # the proof's bound (its condition is 3/2)
