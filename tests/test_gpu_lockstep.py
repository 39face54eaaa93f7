"""The kernels whose warps go through the slots block by block (two-lane
bundles, mixed KS with the FP32 branch) at sizes that leave warps of a block
without rays."""
import numpy as np
import pytest

import oracle_lib as O
from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    import kerrtracecpp2_b200 as kt

    with kt.Renderer(0) as r:
        yield r


@pytest.mark.parametrize("L", [0.0, 1e-5])
@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (17, 1), (65, 1), (33, 7)])
def test_small_bundle_frames_match_oracle(renderer, w, h, L):
    import torch

    d = abi.frame_desc(chart=1, bundles=1, a=0.95, Lambda=L, theta_deg=55.0, width=w, height=h, max_steps=300,
                       flags=abi.KT_FLAG_BUNDLE_FULL_CREEP)
    out = renderer.trace(d)
    torch.cuda.synchronize()
    for k, v in O.trace_port(d, counters=True).items():
        g = out[k].cpu().numpy().view(v.dtype)
        assert np.array_equal(g.view(np.uint8), v.view(np.uint8)), k


@pytest.mark.parametrize("w,h", [(1, 1), (33, 1), (250, 3), (300, 260)])
def test_mixed_ks_sizes(renderer, w, h):
    """Mixed KS frames at the default tolerance (FP32 branch on): reproducible,
    every ray written, and as close to the FP64 frame as the tolerance of the
    mixed tracer at full size (test_gpu_mixed.py): class mismatches below
    1e-4 (none below 10^4 rays), g p50 5e-6."""
    import torch

    kw = dict(chart=0, a=0.7, Q=0.1, theta_deg=70.0, r_obs=50.0, disk_out=15.0, width=w, height=h)
    d = abi.frame_desc(precision=abi.KT_PREC_MIXED, **kw)
    outs = []
    for fill in (0, 255):
        o = renderer.alloc(w * h)
        for v in o.values():
            v.view(torch.uint8).fill_(fill)
        renderer.trace(d, o)
        torch.cuda.synchronize()
        outs.append({k: v.cpu().numpy() for k, v in o.items()})
    for k in outs[0]:
        assert np.array_equal(outs[0][k].view(np.uint8), outs[1][k].view(np.uint8)), k
    ref = renderer.trace(abi.frame_desc(**kw))
    torch.cuda.synchronize()
    oc = ref["outcome"].cpu().numpy()
    miss = int((outs[0]["outcome"] != oc).sum())
    assert miss <= (0 if w * h < 10_000 else 1e-4 * w * h)
    both = (oc == 1) & (outs[0]["outcome"] == 1)
    if both.sum() > 100:
        g = ref["redshift"].cpu().numpy()[both]
        assert np.median(np.abs(outs[0]["redshift"][both] / g - 1)) < 5e-6
