"""The profile's count of launched kernels: camera, resolve, a shade and a trace per round, a check per
iteration of the round loop (its rounds: the depth rounded up to even when the samples are injected at
once, else eight), and one launch that darkens the slots that the caller takes whole."""
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth,wave,body", [(2, 0, 2), (5, 0, 6), (8, 0, 8), (9, 0, 8), (5, 2048, 8)])
@pytest.mark.parametrize("whole", [False, True])
@pytest.mark.parametrize("host_loop", [False, True])
def test_launches(tmp_path, depth, wave, body, whole, host_loop):
    import torch
    s = scenes.cornell(4, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    W, H, spp = 48, 32, 4
    cam = swr.load_camera(s["camera"], W, H)
    samples = torch.empty((W * H, spp, 4), device="cuda") if whole else None
    _, p = sc.render(cam, W, H, spp, depth, seed=1, wave_size=wave, samples=samples, host_loop=host_loop,
                     return_profile=True)
    rounds = p["iterations"]
    assert rounds == p["trace_launches"] and rounds % (8 if host_loop else body) == 0 and rounds > 0
    checks = 0 if host_loop else rounds // body
    assert p["launches"] == 2 + 2 * rounds + checks + (1 if whole else 0)
