"""Images in which most samples reach a light, and images of few pixels with many samples: the resolve
adds the slots of all of them in sample order. Sample counts around its groups of eight and words of 32,
pixel counts around a warp's 32."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(tmp_path, share):
    s = scenes.cornell(4, str(tmp_path))
    d = swr.load_scene(s["scene"], s["basepath"])
    m = d.materials.copy()
    lit = np.random.default_rng(3).random(len(m)) < share
    m["light_source"], m["light_strength"] = lit, np.where(lit, 3.0, 0.0)
    return swr.Scene(swr.SceneData(d.vpos, d.vnrm, d.tri, d.tri_obj, d.obj_first_vertex, m, tri_rank=d.tri_rank,
                                   ranks_exact=d.ranks_exact))


def _ordered_sum(samples, scale):
    acc = np.zeros((samples.shape[0], 3), np.float32)
    for s in range(samples.shape[1]):
        on = samples[:, s, 3] != 0
        acc[on] = acc[on] + samples[on, s, :3]
    return (acc.astype(np.float64) * scale).astype(np.float32)


@pytest.mark.parametrize("spp", [1, 7, 8, 9, 24, 31, 32, 33, 40, 1056])
@pytest.mark.parametrize("share,eye", [(2.0, 0.2), (0.5, 0.2), (2.0, 3.4)])
def test_image_is_the_ordered_sum(tmp_path, spp, share, eye):
    import torch
    sc = _scene(tmp_path, share)
    inv = np.float64(np.float32(1.0) / np.float32(spp))
    for W, H in ((1, 1), (31, 1), (8, 4), (11, 3), (19, 17)):
        cam = swr.make_camera((eye, 0.1, 0.0), (1.0, 0.0), W, H, fov_deg=60.0)
        for mode in (N.MODE_REFERENCE, N.MODE_PHYSICAL):
            samples = torch.full((W * H, spp, 4), float("nan"), device="cuda")
            img = sc.render(cam, W, H, spp, 4, seed=3, mode=mode, samples=samples)
            got = samples.cpu().numpy()
            lit = np.mean(np.any(got[..., :3] != 0, axis=-1))
            assert eye != 0.2 or (lit == 1.0 if share > 1.0 else lit > 0.0)  # from outside: dark pixels too
            assert eye == 0.2 or W * H < 300 or 0.0 < lit < 1.0
            want = _ordered_sum(got, 6.283185307179586 * inv if mode == N.MODE_REFERENCE else inv)
            assert np.array_equal(img.cpu().numpy().reshape(-1, 3), want)
            assert torch.equal(img, sc.render(cam, W, H, spp, 4, seed=3, mode=mode))
        if spp > 100:
            continue
        samples = torch.full((W * H, spp, 4), float("nan"), device="cuda")
        img = sc.render_bdpt(cam, W, H, spp, 4, 3, 4, seed=3, samples=samples).cpu().numpy().reshape(-1, 3)
        assert np.array_equal(img, _ordered_sum(samples.cpu().numpy(), 6.283185307179586 * inv))
