"""The order of a batch's rays (kt_batch_order.h): every chunk's rank against a
sort by (j + 1/2) / F, and its cost by frame sizes, not frames."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import testlibs

SRC = os.path.join(testlibs.TESTS, "kt_batchorder.cpp")
LIB = os.path.join(testlibs.BUILD, "libkt_batchorder.so")


@pytest.fixture(scope="module")
def bo():
    os.makedirs(testlibs.BUILD, exist_ok=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", LIB, SRC], check=True)
    return ctypes.CDLL(LIB)


def _ranks(bo, sizes):
    s = np.asarray(sizes, np.uint64)
    rank = np.full(int((s // 32).sum()), 0xffffffff, np.uint32)
    classes = bo.bo_ranks(len(s), s.ctypes.data_as(ctypes.c_void_p), rank.ctypes.data_as(ctypes.c_void_p))
    return rank, classes


@pytest.mark.parametrize("sizes", [
    [1], [31, 32], [32, 32], [64, 1, 32, 96], [33, 1000, 0x7fff, 64], [3072] * 5, [32 * f for f in range(1, 40)],
    [32 * f for f in (6, 3, 12, 6, 9, 3, 1, 2, 6)], list(np.random.default_rng(1).integers(1, 5000, 60))])
def test_ranks_are_the_sorted_order(bo, sizes):
    rank, classes = _ranks(bo, sizes)
    chunks = [(Fraction(2 * j + 1, 2 * (s // 32)), k, j) for k, s in enumerate(map(int, sizes)) for j in range(s // 32)]
    order = sorted(range(len(chunks)), key=lambda i: chunks[i])
    want = np.empty(len(chunks), np.uint32)
    want[order] = np.arange(len(chunks))
    assert np.array_equal(rank, want)
    assert classes == len({int(s) // 32 for s in sizes} - {0})


def test_many_frames(bo):
    """20,000 frames of two sizes are two classes (a sum over frames would take
    400 million steps here)."""
    rank, classes = _ranks(bo, [256, 64] * 10_000)
    assert classes == 2
    assert np.array_equal(np.sort(rank), np.arange(len(rank)))
