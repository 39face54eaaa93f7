"""kt_exact.cuh on the device it is for: the hardware's reciprocal and root
seeds against the error that the proofs assume, over every significand they
see; quotients, roots, sincos, pow and the exact right-hand sides over the
hard operands of test_exact.py, bit for bit (tests/exact_device.cu)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import test_exact as te
import test_exact_seeds as ts
import testlibs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ed():
    os.makedirs(testlibs.BUILD, exist_ok=True)
    lib = os.path.join(testlibs.BUILD, "libkt_exact_device.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--fmad=false",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared", "-I", testlibs.CSRC, "-o", lib,
                    os.path.join(testlibs.TESTS, "exact_device.cu")], check=True)
    L = ctypes.CDLL(lib)
    P, D, N, I = ctypes.c_void_p, ctypes.c_double, ctypes.c_long, ctypes.c_int
    L.ed_seeds.argtypes = [I, P, P]
    L.ed_quot.argtypes = [N, P, P, P]
    L.ed_values.argtypes = [I, N, P, P]
    L.ed_rhs.argtypes = [I, I, D, D, D, D, N, P, P]
    return L


@pytest.mark.parametrize("root", [0, 1])
def test_seeds_within_the_proofs_bound(ed, root):
    worst, other = ctypes.c_double(), ctypes.c_ulonglong()
    assert ed.ed_seeds(root, ctypes.byref(worst), ctypes.byref(other)) == 0
    print("seed error 2^%.3f" % np.log2(worst.value))
    assert other.value == 0
    assert worst.value <= 2.0 ** -19


def test_quotients_roots_and_functions(ed):
    bad = ctypes.c_ulonglong()
    a, b = ts.quot_operands(4_000_000)
    assert ed.ed_quot(len(a), te._p(a), te._p(b), ctypes.byref(bad)) == 0
    assert bad.value == 0
    x = ts.root_operands(2_000_000)
    assert ed.ed_values(0, len(x), te._p(x), ctypes.byref(bad)) == 0
    assert bad.value == 0
    rng = np.random.default_rng(14)
    x = np.concatenate([rng.uniform(-10, 10, 500_000), te._bits(rng, 500_000, -60, 60),
                        np.abs(te._bits(rng, 500_000, -1022, 1024)), 1.0 + np.arange(-2000, 2000) * 2.0 ** -52,
                        np.arange(-400, 400) * (np.pi / 4), [0.0, -0.0, np.inf, -np.inf, 5e-324]])
    assert ed.ed_values(1, len(x), te._p(x), ctypes.byref(bad)) == 0
    assert bad.value == 0


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("M,a,Q,L", [(1.0, 0.998, 0.0, 0.0), (1.0, 0.0, 0.2, 0.0), (2.5, -1.1, 2.0, 0.0),
                                     (1.0, 0.9, 0.3, 1e-4), (1.0, 0.5, 0.0, -1e-2)])
def test_right_hand_sides(ed, kind, M, a, Q, L):
    if kind == 1 and L != 0.0:
        pytest.skip("the KS chart has no Lambda")
    rng = np.random.default_rng(15 + kind)
    n = 400_000
    y = te._states(rng, n)
    if kind == 1:
        y = np.hstack([rng.uniform(-1, 1, (n, 3)) * np.exp(rng.uniform(-1, 5, (n, 1))),
                       rng.uniform(-2, 2, (n, 3)), -rng.uniform(0.5, 1.5, (n, 1))])
        y[: n // 50, 2] = 0.0
    if kind == 2:
        y = np.hstack([y, rng.uniform(-5, 5, (n, 8))])
    y = np.ascontiguousarray(y)
    for lam in ([1] if L != 0.0 or kind == 1 else [0, 1]):
        out = (ctypes.c_ulonglong * 2)()
        assert ed.ed_rhs(kind, lam, M, a, Q, L, n, te._p(y), out) == 0
        assert out[0] == 0
        assert out[1] < 0.05 * n
