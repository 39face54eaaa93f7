"""bench.py's roofline counts what the kernels execute: below what the FP64 pipe
was measured busy with, and so far below the division-weighted count, which
charges the quotients the cost of divisions that are not there."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
from kerrtracecpp2_b200 import abi  # noqa: E402

# the costs and counters that the headline frame was measured with
COSTS = {"div": 25.93, "div3": 15.5, "sqrt": 27.36, "sincos": 136.64, "pow": 250.74}


def test_headline_frame():
    d = abi.frame_desc(**bench.WORKLOADS["knds_bl_dopri5_720p"])
    n = d.width * d.height
    att = n * (875.5234 - 1.0) / 6.0
    r = bench.roofline_of(d, 0.0, att, COSTS, 34182.65, 38.172)
    # ncu: the FP64 pipe is active in 75% of this kernel's cycles, and an
    # instruction is one or two flops
    assert 0.75 / 2 < r["frac"] < 0.75
    assert r["frac_division_equivalent"] == pytest.approx(0.934, abs=2e-3)
    assert r["achieved"] == pytest.approx(r["flops_per_frame"] / 38.172e-3 / 1e12)


def test_counts():
    assert bench.EXEC_RHS == {True: 808, False: 706}
    d = dict(chart=1, a=0.9, width=10, height=10)
    rk4 = bench.executed_flops(abi.frame_desc(**d), 500.0, 600.0, bench.UNIT_WEIGHTS)
    assert rk4 == pytest.approx((100 + 6000 + 500) * 706 + 600 * (237 + 2 + 1 + 113))
    dp = bench.executed_flops(abi.frame_desc(integrator=1, Lambda=1e-4, **d), 500.0, 600.0, bench.UNIT_WEIGHTS)
    assert dp == pytest.approx((100 + 3600) * 808 + 600 * (256 + 5 + 1 + 113))
    assert bench.executed_flops(abi.frame_desc(chart=0), 1.0, 1.0, bench.UNIT_WEIGHTS) is None
