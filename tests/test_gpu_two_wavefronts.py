"""Renders that run as two concurrent sub-wavefronts (2^20 samples or more and 2^15 triangles or more,
with 2^17 paths in flight or 2^16 triangles): images and samples are those of a single wavefront, into
device and host memory, and a host image does not make the second sub-wavefront wait for the first."""
import ctypes
import time

import numpy as np
import pytest

import master_thesis_b200 as swr
from master_thesis_b200 import _native as N
from master_thesis_b200 import scenes

pytestmark = pytest.mark.gpu


def _scene(tris):
    sd, c = scenes.random_scene(7, tris)
    assert abs(sd.num_triangles - tris) < 2000
    W, H = 256, 256
    return swr.Scene(sd), swr.make_camera(np.array(c["position"]), c["angle"], W, H, fov_deg=40.0), W, H


def _call(sc, cam, W, H, spp, flags, out, samples=None, wave=0):
    import torch
    o = N.RenderOpts(W, H, spp, 6, 5, 0, 0, 1.0, wave, 0, flags | (N.RENDER_SAMPLES_OUT if samples is not None else 0),
                     0, 0, 0)
    N.check(N.lib.swr_render(sc.handle, ctypes.byref(cam), ctypes.byref(o), N.ptr(out), N.ptr(samples),
                             torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("tris", [33_000, 60_000, 90_000])
@pytest.mark.parametrize("wave", [0, 1 << 16, 1 << 17])
def test_two_wavefronts_as_one(tris, wave):
    import torch
    sc, cam, W, H = _scene(tris)
    got = []
    for flags in (N.RENDER_ONE_WAVEFRONT, 0):
        out = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
        smp = torch.empty((H * W, 16, 4), dtype=torch.float32, device="cuda")
        _call(sc, cam, W, H, 16, flags, out, smp, wave)
        _call(sc, cam, W, H, 16, flags, out, None, wave)
        got.append((out, smp))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert int(torch.count_nonzero(got[0][0])) > 0
    pageable = np.full((H, W, 3), np.nan, np.float32)
    pinned = torch.full((H, W, 3), float("nan")).pin_memory()
    _call(sc, cam, W, H, 16, 0, pageable, None, wave)
    _call(sc, cam, W, H, 16, 0, pinned.numpy(), None, wave)
    want = got[0][0].cpu().numpy()
    assert np.array_equal(pageable, want) and np.array_equal(pinned.numpy(), want)


@pytest.mark.parametrize("tris", [33_000, 90_000])
def test_host_image_does_not_serialise_the_wavefronts(tris):
    """One after the other, the halves of the image take half as long again as the whole of it."""
    sc, cam, W, H = _scene(tris)
    out = np.empty((H, W, 3), np.float32)
    best = []
    for flags in (N.RENDER_ONE_WAVEFRONT, 0):
        for _ in range(3):
            _call(sc, cam, W, H, 16, flags, out)
        ts = []
        for _ in range(30):
            t = time.perf_counter()
            _call(sc, cam, W, H, 16, flags, out)
            ts.append(time.perf_counter() - t)
        best.append(min(ts))
    assert best[1] < 1.25 * best[0], best


def test_few_paths_in_flight_stay_one_wavefront():
    """40,000 triangles, 2^16 paths in flight: as two wavefronts the render takes a fifth longer."""
    import torch
    sc, cam, W, H = _scene(40_000)
    out = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
    best = []
    for flags in (N.RENDER_ONE_WAVEFRONT, 0):
        ts = []
        for _ in range(8):
            t = time.perf_counter()
            _call(sc, cam, W, H, 32, flags, out, None, 1 << 16)
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t)
        best.append(min(ts[2:]))
    assert best[1] < 1.08 * best[0], best
