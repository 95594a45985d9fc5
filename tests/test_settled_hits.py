"""Hits whose triangle fails the reference's own slab test: the traversal finds them first, settles
them only when the ray is finished and then traces the ray again with the test on every candidate.
Far from the origin the reference's 1e-4 padding of a box vanishes in the rounding, so that its
boxes of axis-aligned triangles are flat and fail (tmin < tmax is strict): such walls are invisible
to it, and the closest hit is what lies behind them."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200.api import MAT_DTYPE
from helpers import Twin
from oracle import oracle as O


def _walls(at, tilt):
    """Axis-aligned quads (flat boxes) at x = at, at + 2, .. before tilted ones, a light among them."""
    pos, nrm, tri, tobj, first = [], [], [], [], [0]
    for k in range(6):
        flat = k % 2 == 0
        x = at + 2.0 * k
        dx = 0.0 if flat else tilt
        base = first[-1]
        pos += [(x - dx, -8, -8), (x - dx, 8, -8), (x + dx, 8, 8), (x + dx, -8, 8)]
        nrm += [(-1, 0, 0)] * 4
        tri += [(base, base + 1, base + 2), (base, base + 2, base + 3)]
        tobj += [k, k]
        first.append(base + 4)
    mats = np.zeros(6, MAT_DTYPE)
    mats["color"] = 0.7
    mats["diffuse_t"] = mats["reflect_t"] = mats["transparent_t"] = mats["refraction_index"] = 1.0
    mats["light_source"][5] = 1
    mats["light_strength"][5] = 4.0
    return swr.SceneData(np.array(pos, np.float32), np.array(nrm, np.float32), np.array(tri), np.array(tobj),
                         np.array(first), mats)


def _rays(at, n, seed):
    rng = np.random.default_rng(seed)
    o = np.zeros((n, 4), np.float32)
    d = np.zeros((n, 4), np.float32)
    o[:, :3] = rng.uniform((at - 6, -4, -4), (at + 14, 4, 4), (n, 3))
    v = rng.normal(size=(n, 3)) * (1.0, 0.3, 0.3)
    d[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    return o, d


@pytest.mark.parametrize("at", [0.0, 8192.0, 65536.0])
def test_twin_settles_as_the_oracle(at):
    sd = _walls(at, 1.0)
    o, d = _rays(at, 4000, 3)
    otri, od2, ot = O.OracleScene.from_scene_data(sd).trace(o, d)
    for postpone in (False, True):
        tri, d2, t = Twin(sd).trace(o, d, postpone=postpone)
        assert np.array_equal(tri, otri)
        assert np.array_equal(d2.view(np.uint32), od2.view(np.uint32))
        assert np.array_equal(t.view(np.uint32), ot.view(np.uint32))
    hit = otri[otri != 0xFFFFFFFF]
    seen_flat = np.mean((hit // 2) % 2 == 0)  # the flat walls disappear far out
    assert (seen_flat > 0.3) if at == 0.0 else (seen_flat == 0.0)
    assert len(hit) > 1000


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0.0, 8192.0, 65536.0])
@pytest.mark.parametrize("n", [1, 31, 4000])
def test_gpu_queries_settle_as_the_oracle(at, n):
    import torch
    sd = _walls(at, 1.0)
    o, d = _rays(at, n, 4)
    otri, od2, _ = O.OracleScene.from_scene_data(sd).trace(o, d)
    sc = swr.Scene(sd)
    got = sc.trace(torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()).cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:, 0], otri)
    assert np.array_equal(got[:, 2], od2.view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0.0, 8192.0])
def test_gpu_renders_settle_as_the_oracle(at):
    """Camera prefix, bounce rounds, batch and occlusion queries on the same walls."""
    import torch
    sd = _walls(at, 1.0)
    sc = swr.Scene(sd)
    W, H, spp, depth = 24, 18, 8, 5
    cam = swr.make_camera((at - 5.0, 0.5, 0.25), (0.0, 0.0), W, H, fov_deg=60.0)
    samples = torch.zeros((W * H, spp, 4), dtype=torch.float32, device="cuda")
    img = sc.render(cam, W, H, spp, depth, seed=5, samples=samples)
    vi, pi, org = swr.camera_arrays(cam)
    osc = O.OracleScene.from_scene_data(sd)
    ps, pp = O.render_reference(osc, O.camera(vi, pi, org), W, H, spp, depth, 5)
    got = samples.cpu().numpy()
    assert np.array_equal(got[..., 3], ps[..., 3])
    assert np.allclose(got[..., :3], ps[..., :3], rtol=1e-4, atol=1e-7)
    batch = swr.Batch()
    out, = batch.render([dict(scene=sc, cam=cam, width=W, height=H, spp=spp, depth=depth, seed=5)])
    assert torch.allclose(out, img, rtol=1e-5, atol=1e-7)
    bd = sc.render_bdpt(cam, W, H, spp, depth, 3, 4, seed=5).cpu().numpy().reshape(-1, 3)
    _, want = O.render_bdpt(osc, O.camera(vi, pi, org), W, H, spp, depth, 3, 4, 5)
    assert np.allclose(bd, want, rtol=1e-4, atol=1e-6)
