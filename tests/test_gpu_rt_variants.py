"""RayTrace frames by every kernel that the library may choose for them: below and above the triangle
counts and at the image sizes where the choice changes, the frames are the same and the oracle's."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import rt, scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris", [1000, 2040, 3000, 70_000])
@pytest.mark.parametrize("size", [(97, 61), (512, 512), (513, 512), (1024, 1023), (1024, 1024)])
def test_frames_of_all_kernels(tris, size):
    import torch
    sd, c = scenes.random_scene(7, tris)
    sc = swr.Scene(sd)
    W, H = size
    cam = swr.make_camera(np.array(c["position"]), c["angle"], W, H, fov_deg=40.0)
    rgb, rgba = rt.render(sc, cam, W, H, 3, 4)
    assert int(torch.count_nonzero(rgb)) > 0
    for blocks in (5, 6):
        for kw in (dict(), dict(refill=1, shade_batch=1), dict(refill=32, shade_batch=32)):
            a, b = rt.render(sc, cam, W, H, 3, 4, blocks_per_sm=blocks, **kw)
            assert torch.equal(a, rgb) and torch.equal(b, rgba)
    begin = (H // 2) * W
    n = min(W, 97)
    want, want8 = O.rt_render(O.OracleScene.from_scene_data(sd), O.camera(*swr.camera_arrays(cam)), W, H, 3, 4, begin,
                              begin + n)
    got = rgb.reshape(-1, 3)[begin:begin + n].cpu().numpy().astype(np.float64)
    want = np.asarray(want, np.float64).reshape(-1, 3)[:n]
    assert np.all(np.abs(got - want) <= 1e-4 * np.maximum(np.abs(want), 1e-6) + 1e-7)
