"""The work that users of this package give it, as cases that can be timed and compared.

A case is a dict of plain values: a scene (kind, size, geometry seed), the entry point and its
arguments. listed() gives one case per use, draw(rng) another one of the same ranges; prepare()
makes what a program holds before the call (the device scene, camera, rays, parameters), run()
makes the one call, exact() computes the same result in 64-bit floats with plain torch, by testing
every ray against every triangle, where that is cheap enough.

The geometry of a scene is fixed by the case; the seed sets the material colours, the camera, the
rays, the parameters and the random-number key, as a program renders many views of one model.
"""
import atexit
import functools
import math
import shutil
import tempfile

import numpy as np
import torch

import master_thesis_b200 as swr
from master_thesis_b200 import diff, rt, scenes

EXACT_PAIRS = 3e9  # ray-triangle tests that exact() takes on


def listed():
    return [
        # picking and visibility queries of an interactive tool: a few thousand rays, latency counts
        dict(name="query_4k", do="query", scene="random", tris=50_000, geom=3, rays=4_097),
        # bulk closest-hit queries on the benchmark's terrain (its traversal microbenchmark)
        dict(name="query_16m", do="query", scene="terrain", cells=1024, spheres=64, geom=2024, rays=1 << 24),
        # a preview thumbnail of a small model, ragged size, Russian roulette: launches count
        dict(name="thumbnail", do="render", scene="random", tris=5_000, geom=5, width=97, height=61, spp=4, depth=6,
             physical=True, rr_depth=3, wave=0),
        # the Cornell box of the reference's scenes at the benchmark's size, reference estimator
        dict(name="cornell", do="render", scene="cornell", geom=1, width=256, height=256, spp=16, depth=5,
             physical=False, rr_depth=0, wave=0),
        # an ordinary render: a model of 200k triangles with mirrors and glass, ragged image
        dict(name="model", do="render", scene="random", tris=200_000, geom=7, width=641, height=479, spp=16, depth=6,
             physical=True, rr_depth=0, wave=0, mixed=True),
        # the benchmark's workload: 2.4 M triangles, 1920x1080, 64 samples, the whole image in flight
        dict(name="terrain_hd", do="render", scene="terrain", cells=1024, spheres=64, geom=2024, width=1920,
             height=1080, spp=64, depth=8, physical=False, rr_depth=0, wave=1 << 27),
        # the bidirectional tracer with the reference's own renderer settings
        dict(name="bdpt", do="bdpt", scene="cornell", geom=1, width=256, height=256, spp=16, depth=5, light_jumps=5,
             max_depth=5),
        # a RayTrace frame with both denoisers at the reference's settings
        dict(name="rt_frame", do="rt", scene="cornell", geom=1, width=1920, height=1080, spp=13, depth=5, gauss=5),
        # differentiable rendering: image and gradients of a tessellated Cornell box (49k triangles)
        dict(name="diff", do="diff", scene="tess", cells=48, geom=11, width=512, height=512, spp=32, depth=6),
        # a dataset render: many small uneven jobs in one batch
        dict(name="batch", do="batch", scene="random", tris=50_000, geom=7, jobs=64, side=128, spp=16, depth=6),
        # one step of batched inverse rendering: images and gradients of all scenes
        dict(name="inverse", do="inverse", scene="random", tris=50_000, geom=13, jobs=16, side=256, spp=16, depth=5),
        # one frame of an animation: the placements of all objects, then the image
        dict(name="animate", do="animate", scene="tiles", cells=256, spheres=64, geom=2024, width=1920, height=1080,
             spp=4, depth=8),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    do = rng.choice(["query", "query", "render", "render", "render", "bdpt", "rt", "diff", "batch", "inverse",
                     "animate"])
    geom = rng.randrange(1, 10_000)

    def scene(kinds):
        kind = rng.choice(kinds)
        if kind == "random":
            return dict(scene="random", tris=_log(rng, 1_000, 500_000), geom=geom)
        if kind == "terrain":
            return dict(scene="terrain", cells=16 * rng.randrange(8, 65), spheres=rng.randrange(0, 65), geom=geom)
        if kind == "tess":
            return dict(scene="tess", cells=rng.randrange(8, 64), geom=geom)
        return dict(scene="cornell", geom=geom)

    def image(samples, least=2):
        """An image of at most about `samples` camera samples, at least `least` to a pixel."""
        w = _log(rng, 49, 1920)
        h = max(31, int(w * rng.uniform(0.5, 1.0)))
        return dict(width=w, height=h, spp=max(least, min(_log(rng, least, 64), samples // (w * h))))

    if do == "query":
        return dict(do=do, rays=_log(rng, 1_000, 1 << 24), **scene(["random", "terrain", "cornell", "tess"]))
    if do == "render":
        physical = rng.random() < 0.5
        return dict(do=do, depth=rng.randrange(2, 9), physical=physical,
                    rr_depth=rng.choice([0, 3]) if physical else 0, wave=0, mixed=rng.random() < 0.5,
                    **image(1 << 26), **scene(["random", "terrain", "cornell", "tess"]))
    if do == "bdpt":
        return dict(do=do, depth=rng.randrange(2, 7), light_jumps=rng.randrange(1, 7), max_depth=rng.randrange(2, 8),
                    **image(1 << 21), **scene(["random", "cornell", "tess"]))
    if do == "rt":
        return dict(do=do, depth=rng.randrange(4, 7), gauss=rng.choice([0, 3, 5, 9]), **image(1 << 25, least=8),
                    **scene(["random", "terrain", "cornell", "tess"]))
    if do == "diff":
        return dict(do=do, depth=rng.randrange(2, 8), **image(1 << 23), **scene(["random", "tess"]))
    if do == "batch":
        return dict(do=do, scene="random", tris=_log(rng, 5_000, 50_000), geom=geom, jobs=rng.randrange(3, 65),
                    side=rng.randrange(32, 200), spp=rng.randrange(1, 33), depth=rng.randrange(2, 8))
    if do == "inverse":
        return dict(do=do, scene="random", tris=_log(rng, 5_000, 50_000), geom=geom, jobs=rng.randrange(2, 17),
                    side=rng.randrange(48, 300), spp=rng.randrange(1, 17), depth=rng.randrange(2, 7))
    return dict(do=do, scene="tiles", cells=16 * rng.randrange(4, 17), spheres=rng.randrange(4, 65), geom=geom,
                depth=rng.randrange(2, 9), **image(1 << 24))


# ---------------------------------------------------------------------------------------------
# scenes


@functools.lru_cache(maxsize=None)
def _root():
    d = tempfile.mkdtemp(prefix="swr_cases_")
    atexit.register(shutil.rmtree, d, True)
    return d


def _join(objs):
    """SceneData of objects (positions, normals, faces, light strength)."""
    pos, nrm, tri, tobj, first = [], [], [], [], [0]
    mats = np.zeros(len(objs), swr.api.MAT_DTYPE)
    for k, (p, n, f, light) in enumerate(objs):
        pos.append(np.asarray(p, np.float32))
        nrm.append(np.asarray(n, np.float32))
        tri.append(np.asarray(f, np.int64) + first[-1])
        tobj.append(np.full(len(f), k, np.uint32))
        first.append(first[-1] + len(p))
        mats[k]["light_source"] = light > 0
        mats[k]["light_strength"] = light
    mats["color"] = 1.0
    mats["diffuse_t"] = mats["reflect_t"] = mats["transparent_t"] = mats["refraction_index"] = 1.0
    return swr.SceneData(np.concatenate(pos), np.concatenate(nrm), np.concatenate(tri), np.concatenate(tobj),
                         np.array(first, np.uint32), mats)


@functools.lru_cache(maxsize=2)
def _terrain(cells, spheres, geom, tile=16):
    """The terrain of scenes.terrain, made in memory: heightfield tiles, spheres and four lights."""
    rng = np.random.default_rng(geom)
    h = scenes.fbm_heights(cells, geom)
    x = np.linspace(-1.0, 1.0, cells + 1).astype(np.float32)
    n = np.stack([-np.gradient(h.astype(np.float64), x.astype(np.float64), axis=1), np.ones(h.shape),
                  -np.gradient(h.astype(np.float64), x.astype(np.float64), axis=0)], -1)
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    p = np.stack([np.broadcast_to(x[None, :], h.shape), h, np.broadcast_to(x[:, None], h.shape)], -1)
    g = tile + 1
    a = (np.arange(tile)[:, None] * g + np.arange(tile)).reshape(-1)
    face = np.stack([a, a + g, a + 1, a + 1, a + g, a + g + 1], -1).reshape(-1, 3)
    objs = []
    for r in range(0, cells, tile):
        for c in range(0, cells, tile):
            objs.append((p[r:r + g, c:c + g].reshape(-1, 3), n[r:r + g, c:c + g].reshape(-1, 3), face, 0.0))
    sp, sn, sf = scenes.icosphere_mesh(4)
    sf = np.array(sf, np.int64)
    for _ in range(spheres):
        rad = math.exp(rng.uniform(math.log(0.01), math.log(0.1)))
        c = rng.uniform(-0.9, 0.9, 2)
        i, j = (int(round((v + 1) / 2 * cells)) for v in c)
        objs.append((sp * rad + np.array([c[0], h[j, i] + rad, c[1]]), sn, sf, 0.0))
    for _ in range(4):
        c = rng.uniform(-0.6, 0.6, 2)
        q = np.array([(-1, 0, -1), (1, 0, -1), (1, 0, 1), (-1, 0, 1)]) * 0.1 + np.array([c[0], 0.8, c[1]])
        objs.append((q, [(0, -1, 0)] * 4, [(0, 1, 2), (0, 2, 3)], 15.0))
    return _join(objs)


@functools.lru_cache(maxsize=160)
def _random(geom, tris):
    return scenes.random_scene(geom, tris)


@functools.lru_cache(maxsize=8)
def _files(kind, geom, cells, spheres):
    root = tempfile.mkdtemp(dir=_root())
    if kind == "cornell":
        return scenes.cornell(geom, root)
    if kind == "tess":
        return scenes.cornell_tessellated(geom, root, wall_cells=cells, box_cells=max(2, cells * 2 // 3))
    return scenes.terrain(geom, root, cells=cells, spheres=spheres)


def _recolored(data, rng, mixed=False):
    """The scene with other material colours; `mixed`: mirrors and glass among the objects."""
    m = data.materials.copy()
    dark = m["light_source"] == 0
    m["color"][dark] = rng.uniform(0.1, 0.9, (len(m), 3))[dark].astype(np.float32)
    if mixed:
        kind = rng.integers(0, 4, len(m))
        mirror, glass = dark & (kind == 1), dark & (kind == 2)
        m["diffuse_t"][mirror] = 0.3
        m["diffuse_t"][glass] = 0.1
        m["reflect_t"][glass] = 0.4
        m["refraction_index"][glass] = 1.5
    return swr.SceneData(data.vpos, data.vnrm, data.tri, data.tri_obj, data.obj_first_vertex, m,
                         tri_rank=data.tri_rank, ranks_exact=data.ranks_exact)


def _scene(case, rng, k=0):
    """(SceneData, camera position, camera angle) of the case, with the seed's colours and camera."""
    kind = case["scene"]
    if kind == "random":
        tris = case["tris"] if not k else int(1_000 * (case["tris"] / 1_000) ** ((k * 0.618034) % 1.0))
        data, cam = _random(case["geom"] * 1009 + k, tris)
        pos, angle = np.array(cam["position"]), cam["angle"]
    elif kind == "terrain":
        data = _terrain(case["cells"], case["spheres"], case["geom"])
        pos, angle = np.array([0.0, 1.3, 2.2]), (-0.5, -0.35)
    else:
        f = _files(kind, case["geom"], case.get("cells", 0), 0)
        data = swr.load_scene(f["scene"], f["basepath"])
        pos, angle = np.array([3.4, 0.0, 0.0]), (1.0, 0.0)
    pos = pos + rng.uniform(-0.02, 0.02, 3)
    return _recolored(data, rng, case.get("mixed", False)), pos, angle


def _camera(case, pos, angle, w, h):
    return swr.make_camera(pos, angle, w, h, fov_deg=0.0 if case["scene"] in ("terrain", "tiles") else 40.0)


# ---------------------------------------------------------------------------------------------
# what a program holds before the call, and the call


def _jobs(case, rng):
    """Jobs of a batch: scenes of uneven size, images of uneven side and sample count."""
    jobs = []
    for k in range(case["jobs"]):
        data, pos, angle = _scene(case, rng, k)
        side = case["side"] if k % 2 == 0 else max(16, case["side"] // 2)
        jobs.append(dict(scene=swr.Scene(data), cam=_camera(case, pos, angle, side, side), width=side, height=side,
                         spp=case["spp"] if k % 3 == 0 else max(1, case["spp"] // 4), depth=case["depth"],
                         seed=int(rng.integers(1 << 40)), mode=swr.MODE_PHYSICAL))
    return jobs


def _parameters(data, rng):
    albedo = torch.from_numpy(rng.uniform(0.1, 0.9, (data.num_triangles, 3)).astype(np.float32)).cuda()
    m = data.materials
    emission = torch.from_numpy((m["color"] * m["light_strength"][:, None]).astype(np.float32)).cuda()
    return albedo.requires_grad_(), emission.requires_grad_()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    do = case["do"]
    state = dict(case=case, seed=int(seed) * 7919 + 1)
    if do in ("batch", "inverse"):
        jobs = _jobs(case, rng)
        state.update(jobs=jobs, batch=swr.Batch())
        if do == "inverse":
            params = [_parameters(j["scene"].data, rng) for j in jobs]
            state.update(albedo=[p[0] for p in params], emission=[p[1] for p in params],
                         weight=[torch.from_numpy(rng.normal(size=(j["height"], j["width"], 3)).astype(np.float32))
                                 .cuda() for j in jobs])
        return state
    if do == "animate":
        f = _files("tiles", case["geom"], case["cells"], case["spheres"])
        scene = swr.Scene.from_file(f["scene"], f["basepath"])
        xf = scene.transforms()
        moving = slice(len(xf) - 4 - case["spheres"], len(xf) - 4)  # the spheres, one step of a random walk
        xf[moving, :3] += rng.normal(0.0, 0.01, (case["spheres"], 3)).astype(np.float32)
        state.update(scene=scene, placements=xf,
                     cam=_camera(case, np.array([0.0, 1.3, 2.2]), (-0.5, -0.35), case["width"], case["height"]))
        return state
    data, pos, angle = _scene(case, rng)
    state.update(data=data, scene=swr.Scene(data))
    if do == "query":
        o, d = scenes.uniform_rays(case["rays"], data.vpos.min(0), data.vpos.max(0), seed)
        state.update(origin=o, direction=d)
        return state
    w, h = case["width"], case["height"]
    state.update(cam=_camera(case, pos, angle, w, h))
    if do == "diff":
        state["albedo"], state["emission"] = _parameters(data, rng)
        state["weight"] = torch.from_numpy(rng.normal(size=(h, w, 3)).astype(np.float32)).cuda()
    if do == "rt":
        state["params"] = dict(vision_jumps=case["depth"], spp=case["spp"],
                               denoisers=[("GaussDenoiser", case["gauss"], 1.0), ("MedianDenoiser",)])
    return state


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "query":
        return state["scene"].trace(state["origin"], state["direction"])
    if do == "batch":
        return state["batch"].render(state["jobs"])
    if do == "inverse":
        images = diff.render_physical_batch(state["batch"], state["jobs"], state["albedo"], state["emission"])
        grads = torch.autograd.grad(images, state["albedo"] + state["emission"], state["weight"])
        return dict(images=[i.detach() for i in images], grads=grads)
    w, h, scene, cam = case["width"], case["height"], state["scene"], state["cam"]
    if do == "render":
        return scene.render(cam, w, h, case["spp"], case["depth"], seed=state["seed"],
                            mode=swr.MODE_PHYSICAL if case["physical"] else swr.MODE_REFERENCE,
                            rr_depth=case["rr_depth"], rr_survive=0.8 if case["rr_depth"] else 1.0,
                            wave_size=case["wave"])
    if do == "bdpt":
        return scene.render_bdpt(cam, w, h, case["spp"], case["depth"], case["light_jumps"], case["max_depth"],
                                 seed=state["seed"])
    if do == "rt":
        if not case["gauss"]:  # the frame alone: radiance and rgba8 image
            return rt.render(scene, cam, w, h, case["spp"], case["depth"])
        return rt.render_frame(scene, cam, w, h, state["params"])
    if do == "diff":
        image = diff.render_physical(scene, cam, state["albedo"], state["emission"], w, h, case["spp"], case["depth"],
                                     seed=state["seed"])
        albedo, emission = torch.autograd.grad(image, (state["albedo"], state["emission"]), state["weight"])
        return dict(image=image.detach(), albedo=albedo, emission=emission)
    scene.set_transforms(state["placements"])
    return scene.render(cam, w, h, case["spp"], case["depth"], seed=state["seed"])


def _triangles(case):
    kind = case["scene"]
    if kind == "random":
        return case["tris"]
    if kind in ("terrain", "tiles"):
        return 2 * case["cells"] ** 2 + case["spheres"] * 5120 + 8
    return 36 if kind == "cornell" else 10 * case["cells"] ** 2 + 24 * max(2, case["cells"] * 2 // 3) ** 2 + 4


def work(case):
    """Each triangle (corners; corner normals where shading reads them) and ray read once, each
    result written once; one box test per level of a binary tree (24 operations), one triangle test
    (60) and, for camera samples, one shading (200) per ray, one ray per sample."""
    do, tris = case["do"], _triangles(case)
    ray = 60 + 24 * math.ceil(math.log2(tris))
    if do == "query":
        return {"bytes": 36 * tris + case["rays"] * (32 + 16), "flops": case["rays"] * ray}
    if do in ("batch", "inverse"):
        rng, pixels, samples, total = 0, 0, 0, 0
        for k in range(case["jobs"]):
            side = case["side"] if k % 2 == 0 else max(16, case["side"] // 2)
            pixels += side * side
            samples += side * side * (case["spp"] if k % 3 == 0 else max(1, case["spp"] // 4))
            total += case["tris"] if not k else int(1_000 * (case["tris"] / 1_000) ** ((k * 0.618034) % 1.0))
        twice = 2 if do == "inverse" else 1
        return {"bytes": twice * (84 * total + 12 * pixels) + (24 * total if do == "inverse" else 0),
                "flops": twice * samples * (ray + 200)}
    pixels = case["width"] * case["height"]
    samples = pixels * case["spp"]
    if do == "diff":
        return {"bytes": 2 * (84 * tris + 12 * pixels) + 24 * tris, "flops": 2 * samples * (ray + 200)}
    out = 12 if do != "rt" else 4 if case["gauss"] else 16
    moved = 2 * 72 * tris if do == "animate" else 0
    return {"bytes": 72 * tris + out * pixels + moved, "flops": samples * (ray + 200)}


# ---------------------------------------------------------------------------------------------
# the same results in 64-bit floats


def _uniforms(seed, pixel, sample, vertex):
    """Four uniforms per entry: Philox-4x32-10 with counter (pixel, sample, vertex, 0), key = seed."""
    m32 = 0xFFFFFFFF
    c = [pixel & m32, sample & m32, vertex & m32, torch.zeros_like(pixel)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m32) ^ c[1] ^ k0, p1 & m32, ((p0 >> 32) & m32) ^ c[3] ^ k1, p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return [(v >> 8).double() / 16777216.0 for v in c]


def _dot(a, b):
    return (a * b).sum(-1)


class _Plain:
    """A scene whose materials are all diffuse, as 64-bit arrays."""

    def __init__(self, data, device):
        at = lambda a, t=torch.float64: torch.as_tensor(np.asarray(a).astype(np.int64 if t == torch.int64 else np.float64),  # noqa: E731
                                                        device=device, dtype=t)
        corner = at(data.tri, torch.int64)
        pos, nrm = at(data.vpos), at(data.vnrm)
        # the edges are the inputs' 32-bit differences
        v = data.vpos[data.tri]
        self.v0, self.e0, self.e1 = pos[corner[:, 0]], at(v[:, 1] - v[:, 0]), at(v[:, 2] - v[:, 0])
        self.corner, self.normal = pos[corner], nrm[corner]
        self.obj = at(data.tri_obj, torch.int64)
        m = data.materials
        self.color, self.strength = at(m["color"]), at(m["light_strength"])
        self.light = at(m["light_source"], torch.int64) != 0
        self.emission = at(m["color"] * m["light_strength"][:, None])

    def hit(self, o, d):
        """(triangle or -1, t) of the closest hit of each ray."""
        tri = torch.full((len(o),), -1, dtype=torch.int64, device=o.device)
        best = torch.full((len(o),), math.inf, dtype=torch.float64, device=o.device)
        step = max(1, (1 << 23) // len(self.v0))
        for a in range(0, len(o), step):
            oo, dd = o[a:a + step, None], d[a:a + step, None]
            h = torch.linalg.cross(dd, self.e1[None])
            det = _dot(self.e0, h)
            s = oo - self.v0
            u = _dot(s, h) / det
            q = torch.linalg.cross(s, self.e0[None].expand_as(s))
            v = _dot(dd, q) / det
            t = _dot(self.e1, q) / det
            t = torch.where((det.abs() >= 1e-7) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-7), t, math.inf)
            b, i = t.min(1)
            best[a:a + step] = b
            tri[a:a + step] = torch.where(b < math.inf, i, -1)
        return tri, best

    def shading_normal(self, tri, p):
        e0, e1, e2 = self.e0[tri], self.e1[tri], p - self.v0[tri]
        d00, d01, d11, d20, d21 = _dot(e0, e0), _dot(e0, e1), _dot(e1, e1), _dot(e2, e0), _dot(e2, e1)
        den = d00 * d11 - d01 * d01
        v, w = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
        b = torch.stack([1 - v - w, v, w], -1)
        n = (b[..., None] * self.normal[tri]).sum(1)
        return n / n.norm(dim=-1, keepdim=True)


def _hemisphere(n, u1, u2):
    z = 2 * u2 - 1
    r = torch.sqrt((1 - z * z).clamp_min(0))
    v = torch.stack([r * torch.cos(2 * math.pi * u1), r * torch.sin(2 * math.pi * u1), z], -1)
    return torch.where((_dot(v, n) < 0)[:, None], -v, v)


def _first_hits(sc, cam, w, h, depth):
    """Per pixel: the ray and hit after the skipped back faces, and the bounce index of that hit."""
    dev = sc.v0.device
    vi, pi, org = (torch.as_tensor(np.array(a, np.float64), device=dev) for a in (cam.view_inv, cam.proj_inv, cam.origin))
    vi, pi = vi.view(4, 4), pi.view(4, 4)
    k = torch.arange(w * h, device=dev)
    x, y = (k % w).double() + 0.5, (k // w).double() + 0.5
    one = torch.ones_like(x)
    t = (torch.stack([2 * x / w - 1, 2 * y / h - 1, one, one], -1) @ pi)[:, :3]
    t = t / t.norm(dim=-1, keepdim=True)
    d = t @ vi[:3, :3]
    d = d / d.norm(dim=-1, keepdim=True)
    o = org.expand_as(d).clone()
    tri, tt = sc.hit(o, d)
    i = torch.zeros_like(k)
    for _ in range(depth):
        p = o + tt[:, None] * d
        back = (tri >= 0) & (_dot(sc.shading_normal(tri.clamp_min(0), p), d) > 0)
        if not bool(back.any()):
            break
        last = back & (i + 1 >= depth)
        tri = torch.where(last, -1, tri)
        go = torch.nonzero(back & ~last)[:, 0]
        i[go] += 1
        o[go] = p[go] + 0.01 * d[go]
        tri[go], tt[go] = sc.hit(o[go], d[go])
    return o, d, tri, tt, i


def _exact_render(sc, cam, case, seed):
    w, h, spp, depth, physical = case["width"], case["height"], case["spp"], case["depth"], case["physical"]
    dev = sc.v0.device
    first = _first_hits(sc, cam, w, h, depth)
    image = torch.zeros((w * h, 3), dtype=torch.float64, device=dev)
    pixel = torch.arange(w * h, device=dev).repeat_interleave(spp)
    sample = torch.arange(spp, device=dev).repeat(w * h)
    o, d, tri, t, i = (a[pixel] for a in first)
    c = torch.ones((len(pixel), 3), dtype=torch.float64, device=dev)
    for v in range(depth):
        keep = tri >= 0
        pixel, sample, o, d, c, tri, t, i = (a[keep] for a in (pixel, sample, o, d, c, tri, t, i))
        if not len(pixel):
            break
        p = o + t[:, None] * d
        n = sc.shading_normal(tri, p)
        obj = sc.obj[tri]
        front = _dot(n, d) <= 0
        u = _uniforms(seed, pixel, sample, torch.full_like(pixel, v))
        lit = sc.light[obj]
        if physical:
            end = lit
            ns = torch.where(front[:, None], n, -n)
            nd = _hemisphere(ns, u[1], u[2])
            add = c * sc.emission[obj]
            c = c * sc.color[obj] * (2 * _dot(ns, nd))[:, None]
            lit = lit & front
            if case["rr_depth"] and v + 1 >= case["rr_depth"]:
                c = c / 0.8000000119209290
                end = end | (u[3] >= 0.8000000119209290)
        else:
            nd = _hemisphere(n, u[1], u[2])
            c = add = c * sc.color[obj] * _dot(n, nd)[:, None]
            lit = end = lit & front
        image.index_add_(0, pixel[lit], add[lit])
        keep = ~end & (i + 1 < depth)
        pixel, sample, c, i = pixel[keep], sample[keep], c[keep], i[keep] + 1
        o, d = (p + 0.01 * nd)[keep], nd[keep]
        tri, t = sc.hit(o, d)
    return (image * ((1 if physical else 2 * math.pi) / spp)).view(h, w, 3)


def _exact_bdpt(sc, cam, case, seed):
    w, h, spp, vj, lj, md = (case[k] for k in ("width", "height", "spp", "depth", "light_jumps", "max_depth"))
    dev = sc.v0.device
    first = _first_hits(sc, cam, w, h, vj)
    image = torch.zeros((w * h, 3), dtype=torch.float64, device=dev)
    lights = [int(k) for k in torch.nonzero(sc.light)[:, 0]]
    of = [torch.nonzero(sc.obj == k)[:, 0] for k in lights]
    begin = torch.tensor([int(t[0]) for t in of], device=dev)
    count = torch.tensor([len(t) for t in of], device=dev)
    color = sc.color[torch.tensor(lights, device=dev)]
    per = max(1, (1 << 17) // spp)  # pixels at a time
    for p0 in range(0, w * h, per):
        pixel = torch.arange(p0, min(w * h, p0 + per), device=dev).repeat_interleave(spp)
        sample = torch.arange(spp, device=dev).repeat(len(pixel) // spp)
        o, d, tri, t, start = (a[pixel].clone() for a in first)
        i = start.clone()
        size = len(pixel)
        draws = torch.zeros_like(pixel)
        total = torch.zeros((size, 3), dtype=torch.float64, device=dev)
        table = lambda k: torch.zeros((k, size, 3), dtype=torch.float64, device=dev)  # noqa: E731
        vp, vn, vc, lp, lc = table(vj), table(vj), table(vj), table(max(lj, 1)), table(max(lj, 1))
        have_v = torch.zeros((vj, size), dtype=torch.bool, device=dev)
        have_l = torch.zeros((max(lj, 1), size), dtype=torch.bool, device=dev)

        def walk(at, c, o, d, tri, t, i, limit, points, colors, have, normals):
            """Follows the samples `at` until they miss, reach a light's front or the limit; the
            samples that reached a light, with their throughput there."""
            lit_at, lit_c = [], []
            while len(at):
                go = (tri >= 0) & (i < limit)
                at, c, o, d, tri, t, i = (a[go] for a in (at, c, o, d, tri, t, i))
                if not len(at):
                    break
                p = o + t[:, None] * d
                n = sc.shading_normal(tri, p)
                obj = sc.obj[tri]
                u = _uniforms(seed, pixel[at], sample[at], draws[at])
                draws[at] += 1
                nd = _hemisphere(n, u[1], u[2])
                c = c * sc.color[obj] * _dot(n, nd if normals is not None else d)[:, None]
                points[i, at], colors[i, at], have[i, at] = p + 0.01 * n, c, True
                if normals is not None:
                    normals[i, at] = n
                lit = sc.light[obj] & (_dot(n, d) <= 0)
                lit_at.append(at[lit])
                lit_c.append(c[lit])
                keep = ~lit & (i + 1 < limit)
                at, c, o, d, i = at[keep], c[keep], (p + 0.01 * nd)[keep], nd[keep], i[keep] + 1
                tri, t = sc.hit(o, d)
            return torch.cat(lit_at) if lit_at else at, torch.cat(lit_c) if lit_c else None

        every = torch.nonzero(tri >= 0)[:, 0]
        ones = torch.ones((size, 3), dtype=torch.float64, device=dev)
        done = tri < 0
        at, c = walk(every, ones[every], o[every], d[every], tri[every], t[every], i[every], vj, vp, vc, have_v, vn)
        if c is not None:
            total[at] = c
            done[at] = True
        at = torch.nonzero(~done)[:, 0]
        u = []
        for _ in range(4):
            u.append(_uniforms(seed, pixel[at], sample[at], draws[at]))
            draws[at] += 1
        which = (u[0][0] * len(lights)).long().clamp_max(len(lights) - 1)
        # the light point is a 32-bit position: whether a ray from it meets the light's own plane
        # again depends on that rounding and on nothing else
        sr, r2 = torch.sqrt(u[1][0].float()), u[2][0].float()
        one = torch.minimum((u[3][0] * count[which]).long(), count[which] - 1) + begin[which]
        b = torch.stack([1 - sr, sr * (1 - r2), sr * r2], -1)[..., None]
        p = b * sc.corner[one].float()
        p = ((p[:, 0] + p[:, 1]) + p[:, 2]).double()
        n = (b * sc.normal[one]).sum(1)
        n = n / n.norm(dim=-1, keepdim=True)
        lp[0, at], lc[0, at] = p + 0.01 * n, color[which]
        if lj > 1 and len(at):
            nd = _hemisphere(n, u[3][1], u[3][2])
            tri, t = sc.hit(p, nd)
            have_l[0, at] = tri >= 0  # without a hit the light subpath is dropped whole
            walk(at, ones[at], p, nd, tri, t, torch.ones_like(at), lj, lp, lc, have_l, None)
        for a in range(vj):
            for k in range(max(lj, 1)):
                at = torch.nonzero(have_v[a] & have_l[k] & ~done)[:, 0]
                if a + k > md or not len(at):
                    continue
                dd = lp[k, at] - vp[a, at]
                dist = dd.norm(dim=-1)
                dn = dd / dist[:, None]
                free = sc.hit(vp[a, at], dn)[1] > dist
                total[at] += torch.where(free[:, None], vc[a, at] * lc[k, at] * _dot(dn, vn[a, at])[:, None] / md, 0.0)
        image.index_add_(0, pixel, total)
    return (image * (2 * math.pi / spp)).view(h, w, 3)


def exact(case, seed):
    if case["do"] not in ("render", "bdpt") or case.get("mixed"):
        return None  # whole numbers (hits, rgba8 frames), or too many rays and triangles to test all pairs
    rays = 1 if case["do"] == "render" else case["max_depth"]
    if case["width"] * case["height"] * case["spp"] * case["depth"] * rays * _triangles(case) > EXACT_PAIRS:
        return None
    rng = np.random.default_rng(seed)
    data, pos, angle = _scene(case, rng)
    cam = _camera(case, pos, angle, case["width"], case["height"])
    sc = _Plain(data, "cuda")
    render = _exact_render if case["do"] == "render" else _exact_bdpt
    return render(sc, cam, case, int(seed) * 7919 + 1)
