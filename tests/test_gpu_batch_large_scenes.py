"""Batches whose rounds take the one-lane traversal, over scenes below and above the triangle counts at
which single renders choose their kernels: images and gradients of the per-scene calls."""
import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


def test_batch_as_single_renders_and_adjoints():
    import torch
    rng = np.random.default_rng(5)
    jobs = []
    for k, (tris, size, spp) in enumerate([(1000, 128, 8), (90_000, 160, 16), (3000, 64, 33), (200_000, 144, 8)]):
        sd, cam = scenes.random_scene(100 + tris, tris)
        jobs.append(dict(scene=swr.Scene(sd), cam=swr.make_camera(cam["position"], cam["angle"], size, size, fov_deg=40),
                         width=size, height=size, spp=spp, depth=6, seed=int(rng.integers(1 << 30)),
                         mode=swr.MODE_PHYSICAL, rr_depth=3, rr_survive=0.8))
    batch = swr.Batch()
    outs = batch.render(jobs)
    # positive weights: the gradient's terms do not cancel, and its sums agree to the float additions
    dl = [torch.ones((j["height"], j["width"], 3), device="cuda") for j in jobs]
    grads = batch.render_adjoint([dict(j, dl_dimage=g) for j, g in zip(jobs, dl)])
    for j, o, g, (ga, ge) in zip(jobs, outs, dl, grads):
        args = (j["cam"], j["width"], j["height"], j["spp"], j["depth"])
        kw = dict(seed=j["seed"], rr_depth=3, rr_survive=0.8)
        want = j["scene"].render(*args, mode=swr.MODE_PHYSICAL, **kw)
        assert float(want.max()) > 0
        assert torch.allclose(o, want, rtol=1e-5, atol=1e-7)
        wa, we = j["scene"].render_adjoint(*args, g, **kw)
        for a, b in ((ga, wa), (ge, we)):
            a, b = a.double(), b.double()
            assert float(b.norm()) > 0 and float((a - b).norm()) <= 1e-4 * float(b.norm())
