"""The exact right-hand sides' fast forms against their general forms, bit for
bit on the host: shared-reciprocal quotients, sincos without case distinctions,
the unrolled BL right-hand side with and without Lambda (tests/kt_exactcheck.cpp)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import testlibs

SRC = os.path.join(testlibs.TESTS, "kt_exactcheck.cpp")
LIB = os.path.join(testlibs.BUILD, "libkt_exactcheck.so")


@pytest.fixture(scope="module")
def ec():
    os.makedirs(testlibs.BUILD, exist_ok=True)
    heads = [os.path.join(testlibs.CSRC, f) for f in os.listdir(testlibs.CSRC)
             if f.endswith((".h", ".cuh"))]
    if not os.path.exists(LIB) or any(os.path.getmtime(d) > os.path.getmtime(LIB)
                                      for d in heads + [SRC]):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-ffp-contract=off",
                        "-march=x86-64-v3", "-shared", "-o", LIB, SRC], check=True)
    L = ctypes.CDLL(LIB)
    P, D, N = ctypes.c_void_p, ctypes.c_double, ctypes.c_long
    L.ec_quot.argtypes, L.ec_quot.restype = [N, P, P, P], N
    L.ec_sincos.argtypes, L.ec_sincos.restype = [N, P, P], N
    L.ec_bl_rhs.argtypes, L.ec_bl_rhs.restype = [D, D, D, D, ctypes.c_int, N, P, P], N
    L.ec_sqrt.argtypes, L.ec_sqrt.restype = [N, P, P], N
    L.ec_bundle_rhs.argtypes, L.ec_bundle_rhs.restype = [D, D, D, D, ctypes.c_int, N, P, P], N
    L.ec_pow.argtypes, L.ec_pow.restype = [N, P], N
    L.ec_no_event.argtypes, L.ec_no_event.restype = [N, P, P, P], N
    L.ec_ks_rhs.argtypes, L.ec_ks_rhs.restype = [D, D, D, N, P, P], N
    return L


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _bits(rng, n, e_lo, e_hi):
    """Random significands, exponents in [e_lo, e_hi), either sign."""
    u = rng.integers(0, 1 << 52, n, dtype=np.uint64) | (
        rng.integers(1023 + e_lo, 1023 + e_hi, n).astype(np.uint64) << np.uint64(52)) | (
        rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63))
    return u.view(np.float64)


def test_quotients_are_the_ieee_ones(ec):
    rng = np.random.default_rng(3)
    n = 1_000_000
    b = _bits(rng, n, -300, 300)
    a = _bits(rng, n, -400, 400)
    # quotients close to a rounding midpoint, exact quotients, powers of two,
    # zeros, and significands next to 1 and 2
    a[: n // 4] = np.ldexp(rng.integers(1 << 53, 1 << 54, n // 4).astype(np.float64), -53) * b[: n // 4]
    a[n // 4: n // 4 + 1000] = b[n // 4: n // 4 + 1000] * 3.0
    a[-1000:-500], a[-500:] = 0.0, -0.0
    b[1000:2000] = np.ldexp(1.0, rng.integers(-300, 300, 1000))
    b[2000:3000] = 1.0 + np.arange(1000) * 2.0 ** -52
    b[3000:4000] = 2.0 - 2.0 ** -18 - np.arange(1000) * 2.0 ** -52
    b[4000:4100] = 2.0 - 2.0 ** -19
    refused = ctypes.c_long()
    assert ec.ec_quot(n, _p(a), _p(b), ctypes.byref(refused)) == 0
    assert 100 <= refused.value < 2000  # the top 18 bits all ones


def test_sincos_core_is_sincos(ec):
    rng = np.random.default_rng(4)
    x = np.concatenate([rng.uniform(-10, 10, 500_000), _bits(rng, 500_000, -60, 60),
                        np.arange(-400, 400) * (np.pi / 4), np.array([0.0, -0.0, np.inf, -np.inf, np.nan,
                        2.0 ** -27, 2.0 ** 26, -2.0 ** -27, 5e-324])])
    plain = ctypes.c_long()
    # NaN results compare bit for bit as well: both come from the same code
    assert ec.ec_sincos(len(x), _p(x), ctypes.byref(plain)) == 0
    # the uniform half, and the 53 of 120 exponents in [-27, 26) of the other
    assert plain.value > 500_000 * (1 + 52 / 120)


def _states(rng, n):
    y = np.empty((n, 6))
    y[:, 0] = np.where(rng.random(n) < 0.3, rng.uniform(0.5, 3.0, n), np.exp(rng.uniform(0, 6, n)))
    y[:, 1] = rng.uniform(0.01, 3.13, n)
    y[:, 2] = rng.uniform(-2, 2, n)
    y[:, 3] = rng.uniform(-30, 30, n)
    y[:, 4] = -rng.uniform(0.5, 1.5, n)
    y[:, 5] = rng.uniform(-30, 30, n)
    q = n // 50
    y[:q, 1] = np.pi / 2          # the equator
    y[q:2 * q, 1] = rng.uniform(-1e-6, 1e-6, q)  # the pole, and across it
    y[2 * q:3 * q, 1] = rng.uniform(3.14, 3.3, q)
    y[3 * q:4 * q, 3] = -0.0      # an equatorial camera's centre row and column
    y[4 * q:5 * q, 5] = 0.0
    y[5 * q:6 * q, 0] = rng.uniform(-3, 0.5, q)
    y[-6:, 0] = [np.nan, np.inf, 0.0, 1e300, 1e-300, -np.inf]
    y[-12:-6, 2] = [np.nan, np.inf, 1e300, 1e-300, -1e160, 0.0]
    return y


@pytest.mark.parametrize("M,a,Q,L", [
    (1.0, 0.998, 0.0, 0.0), (1.0, 0.0, 0.0, 0.0), (1.0, -0.7, 0.3, 0.0), (2.5, 1.1, 0.0, -0.0),
    (1.0, 0.9, 0.3, 1e-4), (1.0, 0.0, 0.2, 1e-4), (1.0, 0.5, 0.0, -1e-2), (1.0, 0.9, 0.0, 0.3),
    (1.0, 1e-14, 0.0, 0.0), (1.0, 0.9, 0.3, 1e-40), (1.0, 0.5, 3.0, 1e-3)])
def test_bl_rhs_exact_is_bl_rhs(ec, M, a, Q, L):
    y = np.ascontiguousarray(_states(np.random.default_rng(5), 200_000))
    for lam in ([1] if L != 0.0 else [0, 1]):
        refused = ctypes.c_long()
        assert ec.ec_bl_rhs(M, a, Q, L, lam, len(y), _p(y), ctypes.byref(refused)) == 0
        tame = (a == 0.0 or abs(a) >= 2.0 ** -40) and (L == 0.0 or abs(L) >= 2.0 ** -90)
        # in range everywhere but at the states chosen to leave it
        assert refused.value < 0.05 * len(y) if tame else refused.value == len(y)


def _hard_roots():
    """x whose square root lies closest to a rounding midpoint: K^2 + D a
    multiple of 2^52 (2^53), D = +-(K - j) or +-(K + j) with small even j, K a
    53-bit integer (found bit by bit from the lowest)."""
    out = []
    for j in range(2, 200, 2):
        for sg in (-1, 1):
            for t in (-1, 1):
                for mb in (52, 53):
                    for k in (0, 1):
                        for b in range(1, mb + 1):
                            if (k * k + sg * (k + t * j)) % (1 << b):
                                k |= 1 << (b - 1)
                                if (k * k + sg * (k + t * j)) % (1 << b):
                                    break
                        else:
                            for kk in (k, k + (1 << 52)):
                                x = kk * kk + sg * (kk + t * j)
                                if 1 << 52 <= kk < 1 << 53 and x > 0:
                                    out.append(float(x >> 52))
    return np.array(out)


def test_roots_are_the_ieee_ones(ec):
    rng = np.random.default_rng(6)
    hard = _hard_roots()
    g = np.ldexp(rng.integers(1 << 53, 1 << 54, 500_000).astype(np.float64), -53)
    x = np.concatenate([np.abs(_bits(rng, 500_000, -250, 250)), g * g, hard, hard * 4.0, hard * 2.0,
                        1.0 + np.arange(2000) * 2.0 ** -52, 4.0 - np.arange(2000) * 2.0 ** -51,
                        np.arange(1.0, 2000.0) ** 2])
    x = np.ascontiguousarray(x)
    refused = ctypes.c_long()
    assert len(hard) > 500
    assert ec.ec_sqrt(len(x), _p(x), ctypes.byref(refused)) == 0
    assert refused.value < 0.02 * len(x)


@pytest.mark.parametrize("M,a,Q", [(1.0, 0.5, 0.0), (1.0, 0.998, 0.0), (1.0, 0.0, 0.0),
                                   (1.0, -0.7, 0.3), (2.5, 1.1, 2.0), (1.0, 1e-14, 0.1)])
def test_ks_rhs_exact_is_ks_rhs(ec, M, a, Q):
    rng = np.random.default_rng(7)
    n = 200_000
    y = rng.uniform(-1, 1, (n, 7))
    y[:, :3] *= np.exp(rng.uniform(-1, 5, n))[:, None]
    y[:, 3:6] *= 2.0
    y[:, 6] = -rng.uniform(0.5, 1.5, n)
    q = n // 50
    for i, c in enumerate((0, 1, 2, 4)):  # coordinate planes, signed zeros
        y[i * q:(i + 1) * q, c] = np.where(rng.random(q) < 0.5, 0.0, -0.0)
    y[4 * q:5 * q, 2] *= 1e-6
    y[5 * q:6 * q, :2] *= 1e-6  # near the axis
    y[-7:, 0] = [np.nan, np.inf, 1e300, 1e-300, -np.inf, 1e-160, 0.0]
    y[-2:, 1:3] = 0.0
    y[-12:-8, 3] = [np.nan, np.inf, 1e300, 1e-160]
    y = np.ascontiguousarray(y)
    refused = ctypes.c_long()
    assert ec.ec_ks_rhs(M, a, Q, n, _p(y), ctypes.byref(refused)) == 0
    tame = a == 0.0 or abs(a) >= 2.0 ** -40
    assert refused.value < 0.05 * n if tame else refused.value == n


def test_controller_pow_is_pow(ec):
    rng = np.random.default_rng(8)
    x = np.concatenate([rng.uniform(0.5, 2.0, 300_000), np.abs(_bits(rng, 300_000, -1022, 1024)),
                        1.0 + np.arange(-2000, 2000) * 2.0 ** -52, np.sqrt(0.5) + np.arange(-50, 50) * 2.0 ** -53,
                        np.array([0.0, -0.0, -1.0, np.inf, np.nan, 5e-324, 2.0 ** -1022, 1.0, 1.7e308]),
                        np.ldexp(1.0, np.arange(-1000, 1000))])
    assert ec.ec_pow(len(x), _p(np.ascontiguousarray(x))) == 0


@pytest.mark.parametrize("target", [np.pi / 2, 0.0])
def test_quick_event_test_dismisses_no_event(ec, target):
    rng = np.random.default_rng(9)
    n = 1_000_000
    s = np.exp(rng.uniform(-30, 1, n))  # distance from the target, down to rounding
    v = np.empty((n, 6))
    v[:, 4] = np.exp(rng.uniform(-20, 4.6, n))
    for i in (0, 1):
        v[:, i] = target + rng.uniform(-1, 1, n) * s
        v[:, 2 + i] = rng.uniform(-2, 2, n) * s / v[:, 4] * np.exp(rng.uniform(-3, 1.5, n))
    v[:, 5] = target
    v[:100, 0] = target
    v[100:200, 1] = target
    v[200:300, 2] = np.nan
    v[300:400, 3] = np.inf
    q = n // 4  # both ends on one side, as between crossings
    v[-q:, 1] = target + np.abs(v[-q:, 1] - target) * np.sign(v[-q:, 0] - target)
    quick, none = ctypes.c_long(), ctypes.c_long()
    assert ec.ec_no_event(n, _p(np.ascontiguousarray(v)), ctypes.byref(quick), ctypes.byref(none)) == 0
    assert quick.value > 0.5 * none.value  # it is worth its place


@pytest.mark.parametrize("M,a,Q,L", [(1.0, 0.998, 0.0, 0.0), (1.0, 0.0, 0.0, 0.0), (1.0, -0.7, 0.3, 0.0),
                                     (1.0, 0.9, 0.2, 1e-5), (1.0, 0.5, 0.0, -1e-2), (1.0, 1e-14, 0.0, 0.0)])
def test_split_bundle_rhs_exact_is_bundle_rhs(ec, M, a, Q, L):
    rng = np.random.default_rng(10)
    n = 100_000
    y = np.ascontiguousarray(np.hstack([_states(rng, n), rng.uniform(-5, 5, (n, 8))]))
    y[:100, 6:] = 0.0
    for lam in ([1] if L != 0.0 else [0, 1]):
        refused = ctypes.c_long()
        assert ec.ec_bundle_rhs(M, a, Q, L, lam, n, _p(y), ctypes.byref(refused)) == 0
        tame = a == 0.0 or abs(a) >= 2.0 ** -40
        assert refused.value < 0.05 * n if tame else refused.value == n
