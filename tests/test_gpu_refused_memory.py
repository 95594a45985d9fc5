"""A call that the device has no memory for is refused with its own error, and the next call is not."""
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


def test_next_call_after_a_refused_allocation(tmp_path):
    import torch
    s = scenes.cornell(4, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    W = H = 64
    cam = swr.load_camera(s["camera"], W, H)
    want = sc.render(cam, W, H, 4, 5, seed=1)
    # vertex tables of 2^28 samples with 32 slots: 0.4 TB
    with pytest.raises(N.SwrError, match="allocation"):
        sc.render_bdpt(swr.load_camera(s["camera"], 4096, 4096), 4096, 4096, 16, 16, 16, 4, chunk=1 << 28)
    assert torch.equal(sc.render(cam, W, H, 4, 5, seed=1), want)
    batch = swr.Batch()
    job = dict(scene=sc, cam=cam, width=W, height=H, spp=4, depth=5, seed=1)
    image = batch.render([job])[0].clone()
    # 3.4e10 pixels: 1.1 TB of camera records
    big = dict(job, cam=swr.load_camera(s["camera"], 46336, 46336), width=46336, height=46336, spp=1, out=image)
    with pytest.raises(N.SwrError, match="allocation"):
        batch.render([big] * 16)
    assert torch.equal(batch.render([job])[0], image)


def test_chunk_of_too_many_samples_takes_no_memory(tmp_path):
    """2^32 samples at once: refused before any buffer of the chunk (68 GB of slots first) is taken."""
    import torch
    s = scenes.cornell(4, str(tmp_path))
    sc = swr.Scene(swr.load_scene(s["scene"], s["basepath"]))
    cam = swr.load_camera(s["camera"], 1024, 1024)
    out = torch.empty((1024, 1024, 3), device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with pytest.raises(N.SwrError, match="allocation"):
        sc.render_bdpt(cam, 1024, 1024, 4096, 5, 5, 5, chunk=0xFFFFFFFF, out=out)
    assert free - torch.cuda.mem_get_info()[0] < 1 << 30
