"""The KS kernel with several lanes per ray (8 lanes up to 8192 rays, 4 up to
80000, one above), bit for bit against the oracle at the edges of its groups
and ranges."""
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


def _check(got, want):
    for k, w in want.items():
        g = got[k].cpu().numpy().view(w.dtype)
        assert np.array_equal(g.view(np.uint8), w.view(np.uint8)), k


@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (7, 5), (64, 128), (8193, 1), (251, 33)])
@pytest.mark.parametrize("a,Q", [(0.998, 0.0), (0.0, 0.3), (1e-14, 0.0)])
def test_small_frames_match_oracle(renderer, w, h, a, Q):
    import torch

    d = abi.frame_desc(a=a, Q=Q, width=w, height=h, fov_deg=35.0, r_obs=25.0, max_steps=400)
    out = renderer.trace(d)
    torch.cuda.synchronize()
    _check(out, O.trace_port(d, counters=True))


@pytest.mark.parametrize("n", [1, 31, 8192, 8193, 79999, 80000, 80001])
def test_pixel_lists_match_oracle(renderer, n):
    """A list of n pixels of a larger frame; the kernel is chosen by n alone."""
    import torch

    d = abi.frame_desc(a=0.7, Q=0.1, width=401, height=200, theta_deg=75.0, max_steps=300)
    pix = np.random.default_rng(n).permutation(d.width * d.height).astype(np.uint32)[:n]
    out = renderer.trace_pixels(d, torch.from_numpy(pix.view(np.int32)).cuda())
    torch.cuda.synchronize()
    sub = np.arange(n) if n < 20000 else np.arange(0, n, 7)
    want = O.trace_port(d, pix=pix[sub], counters=True)
    _check({k: v[torch.from_numpy(sub).cuda()] for k, v in out.items()}, want)


@pytest.mark.parametrize("integrator", [abi.KT_RK4_DOUBLING, abi.KT_DOPRI5])
def test_rays_that_fail_the_ks_set_up(renderer, integrator):
    """A camera on the axis: every ray goes through the group kernel's
    fallback list to the BL launch; an empty list traces nothing."""
    import torch

    d = abi.frame_desc(a=0.5, width=33, height=21, theta_deg=0.0, integrator=integrator, max_steps=300)
    out = renderer.trace(d)
    torch.cuda.synchronize()
    _check(out, O.trace_port(d, counters=True))
    renderer.trace_pixels(d, torch.empty(0, dtype=torch.int32, device="cuda"))
