"""Register spills of the KS gradient's VJP, from the compiler's listing beside
the object (kerrtracecpp2_b200/_build/*.log): the kernel is out of registers,
and which function spills decides its speed (512 B in the VJP: 10% of a small
frame's gradient)."""
import os
import re

import pytest

from kerrtracecpp2_b200 import build

LOG = os.path.join(build.BUILD, "kt_adjoint.cu.o.log")


def test_ks_gradient_vjp_keeps_its_registers():
    if not os.path.exists(LOG):
        pytest.skip("library built elsewhere: no compiler listing")
    kernel, func, spills = None, None, {}
    for line in open(LOG):
        m = re.search(r"Compiling entry function '(\w+)'", line)
        if m:
            kernel = m.group(1)
        m = re.search(r"Function properties for (\w+)", line)
        if m:
            func = m.group(1)
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m and "k_smoothINS_7ChartKSELb1" in kernel and "sm_vjp_fINS_7ChartKS" in func:
            spills[kernel] = max(map(int, m.groups()))
    assert len(spills) == 2  # blocks of 64 and of 256 threads
    assert max(spills.values()) < 128, spills
