"""Scenes whose rays start with the slab tests on every candidate, because a sixteenth or more of their area
lies in triangles with flat reference boxes, and the same walls beside so much other area that rays start
without them: hits and images are the oracle's either way, also when the objects get there by
set_transforms, with one lane and with eight lanes per ray."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import rt, scenes
from master_thesis_b200.api import MAT_DTYPE
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _scene(at, big):
    """Tilted diffuse wall, flat wall, tilted light; big: and a tilted plane of 400 times their area."""
    pos, nrm, tri, tobj, first = [], [], [], [], [0]
    quads = [(at, 1.0, 8.0, 1.0), (at + 2.0, 0.0, 8.0, 1.0), (at + 4.0, -1.0, 8.0, -1.0)]
    if big:
        quads.append((at - 300.0, 40.0, 280.0, 1.0))
    for k, (x, dx, r, nx) in enumerate(quads):
        b = first[-1]
        pos += [(x - dx, -r, -r), (x - dx, r, -r), (x + dx, r, r), (x + dx, -r, r)]
        nrm += [(nx, 0, 0)] * 4
        tri += [(b, b + 1, b + 2), (b, b + 2, b + 3)]
        tobj += [k, k]
        first.append(b + 4)
    m = np.zeros(len(quads), MAT_DTYPE)
    m["color"] = 0.7
    m["diffuse_t"] = m["reflect_t"] = m["transparent_t"] = m["refraction_index"] = 1.0
    m["light_source"][2], m["light_strength"][2] = 1, 4.0
    return swr.SceneData(np.array(pos, np.float32), np.array(nrm, np.float32), np.array(tri), np.array(tobj),
                         np.array(first), m)


@pytest.mark.parametrize("builder", ["host", "device"])
@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("at", [0.0, 1500.0, 2047.0, 2050.0, 8192.0, 65536.0])
def test_hits_and_images(at, big, builder):
    import torch
    sd = _scene(at, big)
    sc, osc = swr.Scene(sd, builder=builder), O.OracleScene.from_scene_data(sd)
    rng = np.random.default_rng(4)
    n = 30000
    o, d = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    o[:, :3] = rng.uniform((at - 2, -4, -4), (at + 6, 4, 4), (n, 3))
    v = rng.normal(size=(n, 3)) * (1.0, 0.3, 0.3)
    d[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    tri, d2, t = osc.trace(o, d)
    for m in (n, 5000):
        got = sc.trace(torch.from_numpy(o[:m]).cuda(), torch.from_numpy(d[:m]).cuda()).cpu().numpy().view(np.uint32)
        assert np.array_equal(got[:, 0], tri[:m])
        assert np.array_equal(got[:, 2], d2[:m].view(np.uint32)) and np.array_equal(got[:, 3], t[:m].view(np.uint32))
    W, H, spp, depth = 200, 150, 2, 4
    cam = swr.make_camera((at + 3.0, 0.5, 0.25), (1.0, 0.0), W, H, fov_deg=60.0)
    ocam = O.camera(*swr.camera_arrays(cam))
    ps, _ = O.render_reference(osc, ocam, W, H, spp, depth, 5)
    assert 0.2 < ps[..., 3].mean() < 0.9
    want = None
    for how in (dict(), dict(wave_size=4096), dict(static_fetch=True)):
        samples = torch.zeros((W * H, spp, 4), dtype=torch.float32, device="cuda")
        img = sc.render(cam, W, H, spp, depth, seed=5, samples=samples, **how)
        got = samples.cpu().numpy()
        assert np.array_equal(got[..., 3], ps[..., 3])
        assert np.allclose(got[..., :3], ps[..., :3], rtol=1e-4, atol=1e-7)
        want = img if want is None else want
        assert torch.equal(img, want)
    job = dict(scene=sc, cam=cam, width=W, height=H, spp=spp, depth=depth, seed=5)
    for kw in (dict(), dict(wave_size=4096)):
        assert torch.allclose(swr.Batch().render([job], **kw)[0], want, rtol=1e-5, atol=1e-7)
    w, h = 24, 18
    c2 = swr.make_camera((at + 3.0, 0.5, 0.25), (1.0, 0.0), w, h, fov_deg=60.0)
    got = sc.render_bdpt(c2, w, h, 4, 4, 3, 5, seed=5).cpu().numpy().reshape(-1, 3)
    _, bd = O.render_bdpt(osc, O.camera(*swr.camera_arrays(c2)), w, h, 4, 4, 3, 5, 5)
    assert np.allclose(got, bd, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("at", [0.0, 2050.0, 8192.0])
@pytest.mark.parametrize("n", [3000, 30000])
def test_ray_queries_know_no_boxes(at, n):
    """The ray tracing pipeline's closest hit has no slab test: the flat wall is there at any distance."""
    import torch
    sd = _scene(at, False)
    rng = np.random.default_rng(4)
    o, d = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    o[:, :3] = rng.uniform((at - 2, -4, -4), (at + 6, 4, 4), (n, 3))
    v = rng.normal(size=(n, 3)) * (1.0, 0.3, 0.3)
    d[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    tri, t = O.rt_trace(O.OracleScene.from_scene_data(sd), o, d)
    assert np.mean(sd.tri_obj[np.minimum(tri, 5)][tri != 0xFFFFFFFF] == 1) > 0.2
    got = rt.trace(swr.Scene(sd), torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()).cpu().numpy().view(np.uint32)
    hit = tri != 0xFFFFFFFF
    assert np.array_equal(got[:, 0], tri) and np.array_equal(got[hit, 3], t[hit].view(np.uint32))


def _visits(sc, o, d):
    import torch
    counts = torch.zeros((len(o), 2), dtype=torch.int32, device="cuda")
    hits = sc.trace(o, d, counts=counts)
    return hits, int(counts[:, 0].sum())


def test_moved_there_and_back(tmp_path):
    """The Cornell box moved 8,192 units away starts its rays as one that was loaded there: as many nodes are
    visited, a third fewer than with every failed ray traced twice; moved back, as many as at first."""
    import torch
    s = scenes.cornell_tessellated(4, str(tmp_path), wall_cells=12, box_cells=8)
    sc = swr.Scene.from_file(s["scene"], s["basepath"])
    home = sc.transforms()
    lo, hi = sc.data.vpos.min(0), sc.data.vpos.max(0)
    o, d = scenes.uniform_rays(40000, lo, hi, 5)
    hits, visits = _visits(sc, o, d)
    away = home.copy()
    away[:, :3] += 8192.0
    sc.set_transforms(away)
    o2 = o.clone()
    o2[:, :3] += 8192.0
    far, far_visits = _visits(sc, o2, d)
    assert int((far[:, 0] != -1).sum()) < int((hits[:, 0] != -1).sum()) // 2  # the walls are gone
    # loaded there: the same world geometry, packed on the host
    moved = swr.Scene.from_file(s["scene"], s["basepath"])
    moved.set_transforms(away)
    assert torch.equal(_visits(moved, o2, d)[0], far)
    assert far_visits < 1.25 * visits
    sc.set_transforms(home)
    back, back_visits = _visits(sc, o, d)
    assert torch.equal(back, hits) and back_visits == visits


@pytest.mark.parametrize("flat_jobs", [0, 1, 3])
def test_batches_of_flat_and_other_scenes(flat_jobs):
    """The rays of all jobs of a batch start alike, by the jobs' share of flat walls; images and gradients are
    those of each scene alone."""
    import torch
    W, H, spp, depth = 80, 60, 4, 4
    jobs, adjoint = [], []
    for k in range(4):
        at = 8192.0 if k < flat_jobs else 0.0
        sc = swr.Scene(_scene(at, False))
        jobs.append(dict(scene=sc, cam=swr.make_camera((at + 3.0, 0.5, 0.25), (1.0, 0.0), W, H, fov_deg=60.0), width=W,
                         height=H, spp=spp, depth=depth, seed=5 + k, mode=N.MODE_PHYSICAL))
        adjoint.append(dict(jobs[-1], dl_dimage=torch.ones((H, W, 3), device="cuda")))
    for kw in (dict(), dict(wave_size=4096)):
        for j, img in zip(jobs, swr.Batch().render(jobs, **kw)):
            want = j["scene"].render(j["cam"], W, H, spp, depth, seed=j["seed"], mode=N.MODE_PHYSICAL)
            assert want.abs().sum() > 0
            assert torch.allclose(img, want, rtol=1e-5, atol=1e-7)
    for j, got in zip(jobs, swr.Batch().render_adjoint(adjoint)):
        want = j["scene"].render_adjoint(j["cam"], W, H, spp, depth, torch.ones((H, W, 3), device="cuda"),
                                         seed=j["seed"])
        for g, w in zip(got, want):
            assert torch.linalg.norm(g - w) <= 1e-4 * torch.linalg.norm(w)


@pytest.mark.parametrize("at", [0.0, 8192.0])
def test_counted_queries(at):
    """Queries that count their nodes and triangles, few (eight lanes each) and many, find the same hits."""
    import torch
    sc = swr.Scene(_scene(at, False))
    o, d = scenes.uniform_rays(30000, (at - 2, -4, -4), (at + 6, 4, 4), 5)
    want = sc.trace(o, d)
    for n in (30000, 5000):
        counts = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
        assert torch.equal(sc.trace(o[:n], d[:n], counts=counts), want[:n])
        assert int(counts[:, 0].min()) >= 1
