"""Every header that a translation unit of the library or a test-only library
includes is among the files whose change rebuilds it."""
import os
import re

import pytest

import testlibs
from kerrtracecpp2_b200 import build


def _includes(path, seen):
    for name in re.findall(r'^\s*#include "([^"]+)"', open(path).read(), re.M):
        p = os.path.normpath(os.path.join(os.path.dirname(path), name))
        if not os.path.exists(p):
            p = os.path.join(testlibs.CSRC, name)
        if os.path.exists(p) and p not in seen:
            seen.add(p)
            _includes(p, seen)
    return seen


def test_library_headers():
    have = {os.path.join(build.CSRC, h) for h in build.HEADERS} | {
        os.path.join(build.ROOT, "include", h) for h in ("kerrtrace.h", "kerrtrace_cuda_render.h")}
    for src in build.CU_SOURCES + build.CXX_SOURCES:
        assert _includes(os.path.join(build.CSRC, src), set()) <= have, src


@pytest.mark.parametrize("src", ["ktmath_shim.c", "kt_hostcheck.cpp"])
def test_host_check_headers(src, monkeypatch):
    deps = []
    monkeypatch.setattr(testlibs, "_newer", lambda target, d: deps.append((target, list(d))) or False)
    testlibs.build_all()
    have = {os.path.normpath(p) for t, d in deps for p in d}
    assert _includes(os.path.join(testlibs.TESTS, src), set()) <= have
