"""Images written to host memory: every way the wavefront loop can run fills the caller's array with
the device image."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", [dict(), dict(host_loop=True), dict(profile=True), dict(host_loop=True, profile=True)])
def test_host_image_is_the_device_image(tmp_path, how):
    s = scenes.cornell(4, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    W, H = 37, 23
    cam = swr.load_camera(s["camera"], W, H)
    want = sc.render(cam, W, H, 16, 5, seed=2).cpu().numpy()
    assert np.count_nonzero(want) > 0
    out = np.full((H, W, 3), np.nan, np.float32)
    sc.render(cam, W, H, 16, 5, seed=2, out=out, **how)
    assert np.array_equal(out, want)
    part = np.full((100, 3), np.nan, np.float32)
    sc.render(cam, W, H, 16, 5, seed=2, out=part, pixel_begin=200, pixel_count=100, **how)
    assert np.array_equal(part, want.reshape(-1, 3)[200:300])
