"""The interleaved ray order of a batch: every ray of every frame traced once,
the records those of one-frame batches (the same kernels over a frame's own
order), and in FP64 those of single traces, at the edges of its 32-ray chunks."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    import kerrtracecpp2_b200 as kt

    with kt.Renderer(0) as r:
        yield r


@pytest.mark.parametrize("sizes", [
    [(1, 1)], [(1, 1), (31, 1)], [(32, 1), (32, 1)], [(33, 1), (1, 1), (64, 1), (5, 6)],
    [(64, 48), (64, 48), (64, 48)], [(96, 31), (3, 3), (40, 40), (1, 700), (31, 33)]])
@pytest.mark.parametrize("precision", [abi.KT_PREC_FP64, abi.KT_PREC_MIXED])
def test_batch_records_are_the_frames(renderer, sizes, precision):
    import torch

    # tol 1e-9: no FP32 right-hand side, so a ray's result depends on the ray alone
    descs = [abi.frame_desc(a=0.1 + 0.1 * i, width=w, height=h, r_obs=25.0, tol=1e-9, max_steps=400,
                            Lambda=1e-4 if i % 3 == 2 else 0.0, chart=i % 2, precision=precision)
             for i, (w, h) in enumerate(sizes)]
    outs = [renderer.alloc(d.width * d.height) for d in descs]
    for o in outs:
        for v in o.values():
            v.view(torch.uint8).fill_(255)
    b = renderer.batch(descs, outs)
    b.launch()
    torch.cuda.synchronize()
    for d, o in zip(descs, outs):
        one = renderer.alloc(d.width * d.height)
        with_one = renderer.batch([d], [one])
        with_one.launch()
        wants = [one] + ([renderer.trace(d)] if precision == abi.KT_PREC_FP64 else [])
        torch.cuda.synchronize()
        for want in wants:
            for k in want:
                assert np.array_equal(o[k].cpu().numpy().view(np.uint8), want[k].cpu().numpy().view(np.uint8)), k
        with_one.close()
    b.close()
