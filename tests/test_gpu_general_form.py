"""Frames whose parameters the exact quotients do not take (Metric::tame: a, Q
or Lambda tiny but not zero): the general kernels, bit for bit against the
oracle and single traces, and without the cost of a refused exact form."""
import numpy as np
import pytest

import oracle_lib as O
from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu

FRAMES = [
    dict(chart=0, a=0.5, Q=1e-13), dict(chart=0, a=-1e-13, theta_deg=0.0, integrator=1),
    dict(chart=1, a=0.9, Q=0.3, Lambda=4.5e-33), dict(chart=1, a=0.9, Lambda=-1e-40, integrator=1, tol=1e-9),
    dict(chart=1, a=0.95, Q=1e-13, bundles=1, theta_deg=55.0, flags=abi.KT_FLAG_BUNDLE_FULL_CREEP),
]


@pytest.fixture(scope="module")
def renderer():
    import kerrtracecpp2_b200 as kt

    with kt.Renderer(0) as r:
        yield r


def _same(got, want):
    for k, w in want.items():
        assert np.array_equal(got[k].cpu().numpy().view(np.uint8), np.ascontiguousarray(w).view(np.uint8)), k


@pytest.mark.parametrize("size", [(1, 1), (33, 7), (67, 131)])
def test_records_match_oracle_and_batches(renderer, size):
    import torch

    descs = [abi.frame_desc(width=size[0], height=size[1], r_obs=25.0, max_steps=300, **kw) for kw in FRAMES]
    # an ordinary frame in each group as well: the group takes the general kernel
    descs += [abi.frame_desc(width=31, height=9, r_obs=25.0, max_steps=300, **dict(kw, a=0.7, Q=0.1, Lambda=0.0))
              for kw in FRAMES]
    outs = [renderer.alloc(d.width * d.height) for d in descs]
    b = renderer.batch(descs, outs)
    b.launch()
    for d, o in zip(descs, outs):
        one = renderer.trace(d)
        torch.cuda.synchronize()
        _same(one, O.trace_port(d, counters=True))
        _same(o, {k: v.cpu().numpy() for k, v in one.items()})
    b.close()


@pytest.mark.parametrize("kw,inside,outside", [
    (dict(chart=1, integrator=1, tol=1e-9, a=0.9, Q=0.3), dict(Lambda=1e-24), dict(Lambda=4.5e-33)),
    (dict(chart=0, a=0.5), dict(Q=1e-9), dict(Q=1e-13)),
])
def test_general_form_is_not_preceded_by_the_exact_one(renderer, kw, inside, outside):
    """The same rays in both forms.  The general form alone takes 1.2 to 1.6 times
    the exact one's time (the divisions it has more); after a refused exact
    form it took 2.0 to 2.4 times."""
    import torch

    times = []
    for extra in (inside, outside):
        d = abi.frame_desc(width=512, height=400, **kw, **extra)
        out = renderer.trace(d)
        ms = []
        for _ in range(5):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            renderer.trace(d, out)
            e[1].record()
            torch.cuda.synchronize()
            ms.append(e[0].elapsed_time(e[1]))
        times.append(min(ms))
    print("exact %.2f ms, general %.2f ms" % tuple(times))
    assert times[1] < 1.8 * times[0]
