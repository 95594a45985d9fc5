"""One launch that sets the parameters of many scenes against the per-scene calls: triangle and object
counts around the launch's block size, device and host buffers."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["device", "host"])
def test_batch_parameters_as_per_scene(where):
    import torch
    datas = [scenes.random_scene(40 + k, n)[0] for k, n in enumerate((4, 252, 256, 260, 3000))]
    rng = np.random.default_rng(2)
    alb = [rng.uniform(0.05, 0.95, (d.num_triangles, 3)).astype(np.float32) for d in datas]
    em = [rng.uniform(0.5, 9.0, (d.num_objects, 3)).astype(np.float32) for d in datas]
    W, H = 24, 16
    cam = swr.make_camera((4.0, 2.5, 4.0), (-0.75, -0.3), W, H, fov_deg=60.0)
    one = [swr.Scene(d) for d in datas]
    many = [swr.Scene(d) for d in datas]
    give = (lambda a: torch.from_numpy(a).cuda()) if where == "device" else (lambda a: a)
    for s, a, e in zip(one, alb, em):
        s.set_albedo(give(a))
        s.set_emission(give(e))
    batch = swr.Batch()
    batch.set_parameters(many, [give(a) for a in alb], [give(e) for e in em])
    lit = 0
    for a, b in zip(one, many):
        x = a.render(cam, W, H, 64, 4, seed=1, mode=swr.MODE_PHYSICAL)
        assert torch.equal(x, b.render(cam, W, H, 64, 4, seed=1, mode=swr.MODE_PHYSICAL))
        lit += int(torch.count_nonzero(x))
    assert lit > 0
    with pytest.raises(swr.SwrError if hasattr(swr, "SwrError") else Exception):
        batch.set_parameters([], [], [])


def test_batch_parameters_refused_under_capture():
    import torch
    d = scenes.random_scene(7, 64)[0]
    scene, batch = swr.Scene(d), swr.Batch()
    alb = torch.full((d.num_triangles, 3), 0.5, device="cuda")
    em = torch.ones((d.num_objects, 3), device="cuda")
    batch.set_parameters([scene], [alb], [em])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        with pytest.raises(Exception, match="captured"):
            batch.set_parameters([scene], [alb], [em], stream=torch.cuda.current_stream())
        alb.add_(0.0)
    g.replay()
    torch.cuda.synchronize()


def test_batch_parameters_from_two_streams():
    """The second call's table is not written before the first call's launch has read its own."""
    import torch
    datas = [scenes.random_scene(60 + k, 256)[0] for k in range(2)]
    alb = [torch.rand((d.num_triangles, 3), generator=torch.Generator().manual_seed(k)).cuda()
           for k, d in enumerate(datas)]
    em = [torch.full((d.num_objects, 3), 2.0 + k, device="cuda") for k, d in enumerate(datas)]
    W, H = 24, 16
    cam = swr.make_camera((4.0, 2.5, 4.0), (-0.75, -0.3), W, H, fov_deg=60.0)
    one, many = [swr.Scene(d) for d in datas], [swr.Scene(d) for d in datas]
    batch = swr.Batch()
    streams = [torch.cuda.Stream() for _ in datas]
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(20_000_000)  # the first launch waits about 10 ms
    for k in range(2):
        batch.set_parameters([many[k]], [alb[k]], [em[k]], stream=streams[k])
    torch.cuda.synchronize()
    for k in range(2):
        one[k].set_albedo(alb[k])
        one[k].set_emission(em[k])
        x = one[k].render(cam, W, H, 64, 4, seed=1, mode=swr.MODE_PHYSICAL)
        assert torch.count_nonzero(x) > 0
        assert torch.equal(x, many[k].render(cam, W, H, 64, 4, seed=1, mode=swr.MODE_PHYSICAL))
