"""The BL kernels' two instantiations (with and without Lambda) and their
general right-hand side (parameters outside the fast quotients' range), bit
for bit against the oracle."""
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


@pytest.mark.parametrize("integrator", [abi.KT_RK4_DOUBLING, abi.KT_DOPRI5])
@pytest.mark.parametrize("a,Q,L", [(0.0, 0.0, 0.0), (0.998, 0.0, 0.0), (0.9, 0.3, 1e-4),
                                   (0.5, 0.0, -1e-4), (1e-14, 0.2, 0.0), (0.9, 0.3, 1e-40)])
def test_bl_instantiations_match_oracle(renderer, integrator, a, Q, L):
    import torch

    d = abi.frame_desc(chart=abi.KT_CHART_BL, integrator=integrator, a=a, Q=Q, Lambda=L, width=37,
                       height=19, theta_deg=82.0, r_obs=30.0, fov_deg=40.0, max_steps=5000)
    out = renderer.trace(d)
    torch.cuda.synchronize()
    want = O.trace_port(d, counters=True)
    for k, w in want.items():
        got = out[k].cpu().numpy().view(w.dtype)
        assert np.array_equal(got.view(np.uint8), w.view(np.uint8)), k
