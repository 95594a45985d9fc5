"""Launches of few rays give each ray eight lanes (at most 24,000 rays, pixels or paths in flight).
Their hits and images must be those of the one-lane kernels, which larger launches take, and of the
oracle; sizes around the group, warp and grid counts and the switch itself."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import rt, scenes
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LIMIT = 24000


def _scene(name, tmp_path):
    if name == "cornell":
        s = scenes.cornell(4, str(tmp_path))
        return swr.load_scene(s["scene"], s["basepath"])
    return scenes.random_scene(21, 3000)[0]


@pytest.mark.parametrize("name", ["cornell", "random"])
@pytest.mark.parametrize("rule", ["reference", "ray query"])
def test_few_queries_as_many(tmp_path, name, rule):
    import torch
    sd = _scene(name, tmp_path)
    sc = swr.Scene(sd)
    o, d = scenes.uniform_rays(LIMIT + 1, sd.vpos.min(0) - 0.1, sd.vpos.max(0) + 0.1, 5)
    d[::97, 0] = 0.0  # axis-parallel components
    d[::89, 1] = -0.0
    trace = sc.trace if rule == "reference" else (lambda a, b: rt.trace(sc, a, b))
    many = trace(o, d)
    for n in (1, 7, 8, 9, 33, 5920, 5921, 17761, LIMIT):
        assert torch.equal(trace(o[:n].contiguous(), d[:n].contiguous()), many[:n])
    if rule == "reference":
        counts = torch.zeros((2000, 2), dtype=torch.int32, device="cuda")
        assert torch.equal(sc.trace(o[:2000].contiguous(), d[:2000].contiguous(), counts=counts), many[:2000])
        assert int(counts[:, 0].min()) >= 1
        tri, d2, _ = O.OracleScene.from_scene_data(sd).trace(o[:500].cpu().numpy(), d[:500].cpu().numpy())
        got = many[:500].cpu().numpy().view(np.uint32)
        assert np.array_equal(got[:, 0], tri) and np.array_equal(got[:, 2], d2.view(np.uint32))


@pytest.mark.parametrize("name", ["cornell", "random"])
def test_few_pixels_and_paths_as_many(tmp_path, name):
    """Camera prefix (pixel ranges), bounce rounds (paths in flight) and the batch's rounds."""
    import torch
    sc = swr.Scene(_scene(name, tmp_path))
    W, H, spp, depth = 200, 150, 3, 5
    cam = swr.make_camera((3.4, 0.6, 0.1), (1.0, -0.1), W, H, fov_deg=50.0)
    whole = sc.render(cam, W, H, spp, depth, seed=2)  # 30,000 pixels, 90,000 paths
    assert float((whole != 0).float().mean()) > 0.005
    few = sc.render(cam, W, H, spp, depth, seed=2, wave_size=4096)
    assert torch.equal(whole, few)
    flat = whole.reshape(-1, 3)
    for begin, count in ((0, 1), (17, 5921), (29999, 1), (100, LIMIT), (0, LIMIT + 1)):
        assert torch.equal(sc.render(cam, W, H, spp, depth, seed=2, pixel_begin=begin, pixel_count=count),
                           flat[begin:begin + count])
    batch = swr.Batch()
    job = dict(scene=sc, cam=cam, width=W, height=H, spp=spp, depth=depth, seed=2)
    wide = batch.render([job], wave_size=4096)[0].clone()
    assert torch.equal(wide, batch.render([job])[0])
