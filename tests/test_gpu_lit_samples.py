"""The resolve reads only the samples whose lit bit is set: the image must be the ordered float sum
of the samples that the call returns, at sample counts around the bit words, above the count whose
words the host clears, with ragged pixel counts, in both modes and through both entry points."""
import ctypes

import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


def _ordered_sum(samples, scale):
    """[n, spp, 4] -> [n, 3]: flagged samples added one by one in float32, then scaled in double."""
    acc = np.zeros((samples.shape[0], 3), np.float32)
    for s in range(samples.shape[1]):
        on = samples[:, s, 3] != 0
        acc[on] = acc[on] + samples[on, s, :3]
    return (acc.astype(np.float64) * scale).astype(np.float32)


@pytest.mark.parametrize("spp", [1, 2, 31, 32, 33, 100, 1024, 1025])
@pytest.mark.parametrize("mode", [N.MODE_REFERENCE, N.MODE_PHYSICAL])
def test_image_is_the_ordered_sum_of_its_samples(tmp_path, spp, mode):
    import torch
    s = scenes.cornell(2, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    for W, H in ((1, 1), (7, 5), (33, 9)):
        cam = swr.load_camera(s["camera"], W, H)
        samples = torch.full((W * H, spp, 4), float("nan"), dtype=torch.float32, device="cuda")
        img = sc.render(cam, W, H, spp, 5, seed=3, mode=mode, samples=samples).cpu().numpy().reshape(-1, 3)
        got = samples.cpu().numpy()
        assert np.all(np.isfinite(got))
        inv = np.float64(np.float32(1.0) / np.float32(spp))
        want = _ordered_sum(got, 6.283185307179586 * inv if mode == N.MODE_REFERENCE else inv)
        assert np.array_equal(img, want)
        plain = sc.render(cam, W, H, spp, 5, seed=3, mode=mode).cpu().numpy().reshape(-1, 3)
        assert np.array_equal(img, plain)
        profiled = sc.render(cam, W, H, spp, 5, seed=3, mode=mode, profile=True).cpu().numpy().reshape(-1, 3)
        assert np.array_equal(img, profiled)
        out = torch.full((H, W, 3), float("nan"), dtype=torch.float32, device="cuda")
        o = N.RenderOpts(W, H, spp, 5, 3, mode, 0, 1.0, 0, 0, 0, 0, 0, 0)
        N.check(N.lib.swr_render_noalloc(sc.handle, ctypes.byref(cam), ctypes.byref(o), N.ptr(out), None,
                                         torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert np.array_equal(img, out.cpu().numpy().reshape(-1, 3))
    assert spp < 30 or np.count_nonzero(img) > 0


def test_tiny_queue_reinjects_over_many_rounds(tmp_path):
    """4096 paths in flight of 30 k samples: injected indices go through the sample division often."""
    s = scenes.cornell(2, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    W, H = 31, 29
    cam = swr.load_camera(s["camera"], W, H)
    for spp in (1, 3, 33):
        a = sc.render(cam, W, H, spp, 5, seed=9)
        b = sc.render(cam, W, H, spp, 5, seed=9, wave_size=4096)
        assert bool((a == b).all())
