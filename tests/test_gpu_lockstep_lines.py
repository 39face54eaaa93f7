"""Mixed KS frames with the FP32 branch around the line above which the kernel's
blocks go through the slots together (192 rays per SM), with warps and whole
blocks of the launch left without rays: every record written, reproducible, and
as close to the FP64 frame as the mixed tracer is at full size."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,beyond", [(192, -1), (192, 0), (192, 1), (256, 33), (384, 0)])
def test_mixed_ks_around_the_lockstep_line(per_sm, beyond):
    import torch

    import kerrtracecpp2_b200 as kt

    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    w = 251
    h = -(-n // w)
    kw = dict(chart=0, a=0.7, Q=0.1, theta_deg=70.0, r_obs=50.0, disk_out=15.0, width=w, height=h)
    pix = torch.arange(n, dtype=torch.int32, device="cuda")
    with kt.Renderer(0) as r:
        outs = []
        for fill in (0, 255):
            o = r.alloc(n)
            for v in o.values():
                v.view(torch.uint8).fill_(fill)
            r.trace_pixels(abi.frame_desc(precision=abi.KT_PREC_MIXED, **kw), pix, out=o)
            torch.cuda.synchronize()
            outs.append({k: v.cpu().numpy() for k, v in o.items()})
        ref = {k: v.cpu().numpy() for k, v in r.trace_pixels(abi.frame_desc(**kw), pix).items()}
    for k in ref:
        assert np.array_equal(outs[0][k].view(np.uint8), outs[1][k].view(np.uint8)), k
    # the bounds of test_gpu_mixed.py: classes 1e-4, g p50 5e-6
    assert (outs[0]["outcome"] != ref["outcome"]).sum() <= 1e-4 * n
    both = (ref["outcome"] == 1) & (outs[0]["outcome"] == 1)
    assert both.sum() > 1000
    assert np.median(np.abs(outs[0]["redshift"][both] / ref["redshift"][both] - 1)) < 5e-6
