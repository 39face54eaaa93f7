"""The KS kernel's lanes per ray change at rays per SM (8 lanes up to 90, 4 up to
540, one above): pixel lists on both sides of each line, bit for bit against
the oracle."""
import numpy as np
import pytest

import oracle_lib as O
from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [90, 540])
@pytest.mark.parametrize("beyond", [0, 1])
def test_lists_at_the_lines_match_oracle(per_sm, beyond):
    import torch

    import kerrtracecpp2_b200 as kt

    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    w = 401
    d = abi.frame_desc(a=0.7, Q=0.1, width=w, height=n // w + 2, theta_deg=75.0, max_steps=300)
    pix = np.random.default_rng(n).permutation(d.width * d.height).astype(np.uint32)[:n]
    with kt.Renderer(0) as r:
        out = r.trace_pixels(d, torch.from_numpy(pix.view(np.int32)).cuda())
        torch.cuda.synchronize()
        sub = np.unique(np.concatenate([np.arange(0, n, 7), np.arange(n - 40, n)]))
        want = O.trace_port(d, pix=pix[sub], counters=True)
        for k, v in want.items():
            got = out[k].cpu().numpy()[sub].view(v.dtype)
            assert np.array_equal(got.view(np.uint8), v.view(np.uint8)), k
