"""Gradient kernels of large frames (rays taken 256 to a block) against the same
pixels in lists short enough for the 64-thread kernels, at ragged sizes just
above the line between them."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(chart=0, a=0.7, r_obs=20.0), dict(chart=1, a=0.7, Lambda=1e-4, r_obs=20.0),
    dict(chart=1, integrator=1, a=0.7, r_obs=20.0, tol=1e-8),
    dict(chart=1, bundles=1, a=0.95, theta_deg=60.0, r_obs=20.0, max_steps=400)])
@pytest.mark.parametrize("extra", [0, 1, 255])
def test_wide_blocks_give_the_listed_pixels_gradient(kw, extra):
    import torch

    import kerrtracecpp2_b200 as kt

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 256 * sms + extra
    w = 97
    d = abi.frame_desc(width=w, height=-(-n // w), **kw)
    size = d.width * d.height
    cot = torch.ones(size, dtype=torch.float64, device="cuda")
    with kt.Renderer(0) as r:
        pix = torch.arange(n, dtype=torch.int32, device="cuda")
        out, ref = r.alloc(size), r.alloc(size)
        for o in (out, ref):
            for v in o.values():
                v.view(torch.uint8).fill_(255)
        grad, _ = r.vjp(d, cot, cot, out=out, pix=pix)
        parts = [r.vjp(d, cot, cot, out=ref, pix=p.contiguous())[0] for p in pix.split(16000)]
        torch.cuda.synchronize()
    for k in out:  # every listed pixel's record, and no other written
        assert torch.equal(out[k].view(torch.uint8), ref[k].view(torch.uint8)), k
    # the same contributions, summed in another order: at most n additions of
    # rounding 2^-53 each, relative to the sum of the magnitudes (bounded
    # through the parts' cancellation by 1e4)
    want = np.sum(parts, axis=0)
    np.testing.assert_allclose(grad, want, rtol=1e4 * n * 2.0 ** -53, atol=1e-300)
