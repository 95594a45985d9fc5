"""Lists of parameter jobs that are not one entry per scene: a scene named more than once keeps its last
entry, lists of different lengths are refused, and so is an empty one."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import diff, scenes

pytestmark = pytest.mark.gpu
W, H = 24, 16


def _image(scene, cam):
    return scene.render(cam, W, H, 64, 4, seed=1, mode=swr.MODE_PHYSICAL)


@pytest.mark.parametrize("where", ["device", "host"])
@pytest.mark.parametrize("tris", [4, 3000])
def test_a_scene_named_twice_keeps_its_last_entry(where, tris):
    import torch
    d = scenes.random_scene(31, tris)[0]
    cam = swr.make_camera((4.0, 2.5, 4.0), (-0.75, -0.3), W, H, fov_deg=60.0)
    rng = np.random.default_rng(6)
    many, one, batch = swr.Scene(d), swr.Scene(d), swr.Batch()
    give = (lambda a: torch.from_numpy(a).cuda()) if where == "device" else (lambda a: a)
    for _ in range(12):
        # 48 entries of one scene: the blocks of all of them are resident at once
        alb = [give(rng.uniform(0.05, 0.95, (d.num_triangles, 3)).astype(np.float32)) for _ in range(48)]
        em = [give(rng.uniform(0.5, 9.0, (d.num_objects, 3)).astype(np.float32)) for _ in range(48)]
        batch.set_parameters([many] * 48, alb, em)
        one.set_albedo(alb[-1])
        one.set_emission(em[-1])
        x = _image(one, cam)
        assert torch.equal(_image(many, cam), x)
    assert int(torch.count_nonzero(x)) > 0


def test_lists_of_different_lengths():
    import torch
    d = scenes.random_scene(32, 64)[0]
    s = [swr.Scene(d), swr.Scene(d)]
    alb = [torch.full((d.num_triangles, 3), 0.25 + 0.25 * k, device="cuda") for k in range(3)]
    em = [torch.full((d.num_objects, 3), 2.0 + k, device="cuda") for k in range(3)]
    batch = swr.Batch()
    with pytest.raises(ValueError, match="2 scenes"):
        batch.set_parameters(s, alb, em[:2])
    with pytest.raises(ValueError, match="2 scenes"):
        batch.set_parameters(s, alb[:2], em[:1])
    with pytest.raises(N.SwrError, match="empty batch"):
        batch.set_parameters([], [], [])
    # the differentiable batch passes over parameters beyond its jobs
    cam = swr.make_camera((4.0, 2.5, 4.0), (-0.75, -0.3), W, H, fov_deg=60.0)
    jobs = [dict(scene=x, cam=cam, width=W, height=H, spp=8, depth=3) for x in s]
    a = diff.render_physical_batch(batch, jobs, alb, em)
    b = diff.render_physical_batch(batch, jobs, alb[:2], em[:2])
    assert len(a) == len(b) == 2 and all(torch.equal(x, y) for x, y in zip(a, b))
    with pytest.raises((ValueError, IndexError)):
        diff.render_physical_batch(batch, jobs, alb[:1], em[:1])


def test_table_is_not_overwritten_while_its_launch_waits():
    """The first call's launch waits for room on a GPU that closest-hit queries fill, its table already
    copied; the second call, on another stream, must not copy its own over it. All scenes are of one size,
    so that whichever table a launch reads fits them."""
    import torch
    datas = [scenes.random_scene(60 + k, 256)[0] for k in range(2)]
    alb = [torch.rand((d.num_triangles, 3), generator=torch.Generator().manual_seed(k)).cuda()
           for k, d in enumerate(datas)]
    em = [torch.full((d.num_objects, 3), 2.0 + k, device="cuda") for k, d in enumerate(datas)]
    assert alb[0].shape == alb[1].shape and em[0].shape == em[1].shape
    one, many = [swr.Scene(d) for d in datas], [swr.Scene(d) for d in datas]
    busy = swr.Scene(scenes.random_scene(9, 100_000)[0])
    o, d = scenes.uniform_rays(1 << 22, busy.data.vpos.min(0), busy.data.vpos.max(0), 5)
    hits = torch.empty((1 << 22, 4), dtype=torch.int32, device="cuda")
    batch = swr.Batch()
    batch.set_parameters(many, alb[::-1], em[::-1])  # the buffers exist before the queries run
    filler, a, b = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for _ in range(8):
        busy.trace(o, d, out=hits, stream=filler)
    done.record(filler)
    batch.set_parameters([many[0]], [alb[0]], [em[0]], stream=a)
    batch.set_parameters([many[1]], [alb[1]], [em[1]], stream=b)
    queued_behind_the_queries = not done.query()
    torch.cuda.synchronize()
    assert queued_behind_the_queries
    cam = swr.make_camera((4.0, 2.5, 4.0), (-0.75, -0.3), W, H, fov_deg=60.0)
    for k in range(2):
        one[k].set_albedo(alb[k])
        one[k].set_emission(em[k])
        x = _image(one[k], cam)
        assert int(torch.count_nonzero(x)) > 0 and torch.equal(x, _image(many[k], cam))
