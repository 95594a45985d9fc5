"""The grid of a wide node's planes: every child's planes lie on the levels that the traversal decodes and
do not cut into the child's box, for boxes of all sizes and places. The levels are compared in 64 bits,
whose rounding of the difference to the origin and of the sum is the only tolerance: 2^-52 of the larger
of the two, far below the margin (2^-16 of the extent) by which the builders enlarge every box."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from helpers import ROOT

N = 200_000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plane_grid") / "plane_grid.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    "-o", so, os.path.join(ROOT, "tests", "native", "plane_grid.cpp")], check=True)
    return ctypes.CDLL(so)


def _grid(lib, lo, hi, clo, chi):
    a = [np.ascontiguousarray(x, np.float32) for x in (lo, hi, clo, chi)]
    n = len(a[0])
    out = [np.empty(n, t) for t in (np.float32, np.int32, np.uint32, np.uint32, np.float32, np.float32)]
    lib.plane_grid_test(ctypes.c_uint64(n), *[ctypes.c_void_p(x.ctypes.data) for x in a + out])
    return a, out


def _check(lib, lo, ext):
    rng = np.random.default_rng(1)
    lo = np.asarray(lo, np.float32)
    hi = np.maximum((lo.astype(np.float64) + ext).astype(np.float32), lo)
    f = np.sort(rng.random((2, len(lo))), axis=0)
    f[:, ::5] = (f[:, ::5] > 0.5)  # children that touch the node's ends
    f = np.sort(f, axis=0)
    span = hi.astype(np.float64) - lo
    clo, chi = (np.clip((lo + f[k] * span).astype(np.float32), lo, hi) for k in (0, 1))
    (lo, hi, clo, chi), (p, e, qb, qa, lb, la) = _grid(lib, lo, hi, clo, chi)
    assert np.all(np.isfinite(p)) and np.all((e >= -126) & (e <= 127))
    level = lambda q: np.where(q < 128, 128.0 + q, 256.0 + 2.0 * (q.astype(np.float64) - 128.0))
    assert np.array_equal(level(qb), lb) and np.array_equal(level(qa), la)
    assert np.all(qb <= 255) and np.all(qa <= 255) and np.all(qb <= qa)
    unit = np.ldexp(1.0, e)
    p64 = p.astype(np.float64)
    below, above = p64 + lb * unit, p64 + la * unit
    tol = 2.0 ** -52 * np.maximum(np.abs(p64), np.maximum(np.abs(clo), np.abs(chi)).astype(np.float64))
    assert np.all(below <= clo + tol)
    assert np.all(above >= chi - tol)
    # not looser than one cell of the coarse half: two units, and the origin's rounding down
    slack = 2.0 * unit + np.spacing(np.abs(p).astype(np.float32)).astype(np.float64)
    assert np.all(clo - below <= slack + tol) and np.all(above - chi <= slack + tol)
    # the unit is the smallest that covers the node, or one step above where the origin's rounding asks it
    far = span < 1e-3 * np.abs(lo)
    big = ~far & (span > 382.0 * 2.0 ** -125)
    assert np.all(unit[big] < 4.0 * span[big] / 382.0)


def test_boxes_of_a_scene(lib):
    rng = np.random.default_rng(2)
    _check(lib, rng.uniform(-3.0, 3.0, N), np.exp(rng.uniform(np.log(1e-6), np.log(6.0), N)))


def test_extents_at_powers_of_two(lib):
    """Extents of just 382 units, where the unit changes, and their float neighbours."""
    e = np.repeat(np.arange(-60, 60), 5)
    at = np.ldexp(382.0, e).astype(np.float32)
    step = np.tile([-2, -1, 0, 1, 2], 120)
    ext = (at.view(np.int32) + step).view(np.float32)
    for lo in (0.0, 1.0, -1.0, -191.0):
        _check(lib, np.full(len(ext), lo), ext.astype(np.float64))


@pytest.mark.parametrize("size,place", [(1e-30, 0.0), (1e-12, 1.0), (1e-5, 1e4), (1.0, 65536.0), (1e-3, 1e7),
                                        (1e9, 1e9), (1e18, 0.0), (1e18, 1e18)])
def test_tiny_huge_and_far_boxes(lib, size, place):
    rng = np.random.default_rng(3)
    _check(lib, rng.uniform(-1.0, 1.0, N) * place, size * rng.random(N))


def test_flat_boxes(lib):
    """No extent: the planes enclose the point."""
    rng = np.random.default_rng(4)
    for s in (0.0, 1e-20, 1.0, 1e6):
        _check(lib, rng.uniform(-1.0, 1.0, 1000) * s, np.zeros(1000))
