"""A batch of thousands of small frames: tables of hundreds of kilobytes are on
the device before the ray order is made from them."""
import numpy as np
import pytest

from kerrtracecpp2_b200 import abi

pytestmark = pytest.mark.gpu


def test_thousands_of_frames_have_the_single_frames_records():
    import torch

    import kerrtracecpp2_b200 as kt

    kinds = [abi.frame_desc(a=0.1 * i, width=8 + i, height=4 + 3 * i, r_obs=20.0, max_steps=200) for i in range(9)]
    n = 20_000
    with kt.Renderer(0) as r:
        want = []
        for d in kinds:
            w = r.trace(d)
            torch.cuda.synchronize()
            want.append({k: v.cpu().numpy() for k, v in w.items()})
        descs = [kinds[i * i % 9] for i in range(n)]
        sizes = [d.width * d.height for d in descs]
        at = np.concatenate([[0], np.cumsum(sizes)])
        whole = r.alloc(int(at[-1]))
        for v in whole.values():
            v.view(torch.uint8).fill_(255)
        b = r.batch(descs, [{k: v[at[i]:at[i + 1]] for k, v in whole.items()} for i in range(n)])
        b.launch()
        torch.cuda.synchronize()
        got = {k: v.cpu().numpy() for k, v in whole.items()}
        b.close()
    for k in got:
        expect = np.concatenate([want[i * i % 9][k] for i in range(n)])
        assert np.array_equal(got[k].view(np.uint8), expect.view(np.uint8)), k
