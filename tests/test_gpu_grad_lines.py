"""The lines between which gradient rays go 256 to a block: the same rays on both
sides of them, and single rays' contributions (a cotangent of one pixel), bit for
bit."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu

KINDS = {
    "ks": (256, dict(chart=0, a=0.7, r_obs=20.0)),
    "rk4": (1024, dict(chart=1, a=0.7, Lambda=1e-4, r_obs=20.0)),
    "dopri5": (1024, dict(chart=1, integrator=1, a=0.7, r_obs=20.0, tol=1e-8)),
    "rk4_upper": (2048, dict(chart=1, a=0.7, Lambda=1e-4, r_obs=20.0)),
    "bundle": (256, dict(chart=1, bundles=1, a=0.95, theta_deg=60.0, r_obs=20.0, max_steps=400)),
}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("beyond", [-1, 0, 1, 255])
def test_single_rays_contribute_the_same_in_either_block(kind, beyond):
    import torch

    import kerrtracecpp2_b200 as kt

    per_sm, kw = KINDS[kind]
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    w = 397
    d = abi.frame_desc(width=w, height=-(-n // w), **kw)
    size = d.width * d.height
    with kt.Renderer(0) as r:
        pix = torch.arange(n, dtype=torch.int32, device="cuda")
        out = r.alloc(size)
        for v in out.values():
            v.view(torch.uint8).fill_(255)
        ones = torch.ones(size, dtype=torch.float64, device="cuda")
        r.vjp(d, ones, ones, out=out, pix=pix)
        # the whole frame's records: the smooth forward's
        want = r.trace(abi.frame_desc(precision=abi.KT_PREC_SMOOTH, width=d.width, height=d.height, **kw))
        torch.cuda.synchronize()
        for k in out:
            assert torch.equal(out[k][:n].view(torch.uint8), want[k][:n].view(torch.uint8)), k
            assert bool((out[k][n:].view(torch.uint8) == 255).all()), k
        hits = torch.nonzero(out["outcome"][:n] == 1).flatten()
        for p in {int(hits[0]), int(hits[len(hits) // 2]), int(hits[-1]), n - 1}:
            cot = torch.zeros(size, dtype=torch.float64, device="cuda")
            cot[p] = 1.0
            many, _ = r.vjp(d, cot, cot, pix=pix)
            alone, _ = r.vjp(d, cot, cot, pix=torch.tensor([p], dtype=torch.int32, device="cuda"))
            assert np.array_equal(np.asarray(many), np.asarray(alone)), p
