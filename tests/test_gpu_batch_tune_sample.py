"""The autotuner's sample: chunks of 32 rays as the launch takes them (8 x 4
pixel blocks of the centre-out order), spread over all frames of the group."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,fraction", [(1, 0.25), (3, 0.25), (4, 0.25), (4, 1.0)])
def test_sample_is_of_the_launch_order(frames, fraction):
    import torch

    import kerrtracecpp2_b200 as kt

    w, h = 72, 40  # 90 blocks a frame
    with kt.Renderer(0) as r:
        descs = [abi.frame_desc(a=0.3 + 0.1 * i, width=w, height=h, r_obs=25.0) for i in range(frames)]
        outs = [r.alloc(w * h) for _ in descs]
        for o in outs:
            o["outcome"].fill_(255)
        b = r.batch(descs, outs, options=abi.batch_options(autotune=True, tune_fraction=fraction, tune_reps=1))
        torch.cuda.synchronize()
        (g,) = b.groups()
        counts = []
        for o in outs:
            blocks = (o["outcome"].cpu().numpy() != 255).reshape(h // 4, 4, w // 8, 8).sum(axis=(1, 3))
            assert set(np.unique(blocks)) <= {0, 32}
            counts.append(int((blocks == 32).sum()))
        b.close()
    assert 32 * sum(counts) == g["sample_rays"]
    # an even share of each frame: the spread's discrepancy is a few chunks
    assert max(abs(c - 90 * fraction) for c in counts) <= (0 if fraction == 1.0 else 6)
