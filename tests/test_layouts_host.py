"""The MIXED form on the three field layouts (planes, row pairs, cells), built
for the host: the second differences a layout stores are the ones the others
form on the spot, so maps, guard flags and state cotangents agree bit for bit,
as do the four-tap passes from any of them with each other;
and the tap cotangents scattered by cells (with the copies of the region around
the observer) and gathered through the second differences' transpose equal the
ones scattered tap by tap. Odd, non-cubic and very small grids, rays that wrap
around the box, and footprints inside and across the region's edge."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import srt_fields

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    if not os.path.isfile(os.path.join(cuda_inc, "cuda_fp16.h")):
        pytest.skip("CUDA headers not found")
    out = str(tmp_path_factory.mktemp("layout") / "liblayout.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + os.path.join(ROOT, "snapshot-raytracer_gb300", "csrc"), "-I" + cuda_inc,
                        os.path.join(ROOT, "tests", "layout_shim.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    L = ctypes.CDLL(out)
    P, I, Q = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    L.layout_maps.argtypes = [P, I, I, I, Q, Q, I, P, P]
    L.scatter_pair.argtypes = [P, I, I, I, Q] + [P] * 6
    L.layout_vjp.argtypes = [P, I, I, I, I] + [P] * 9 + [I]
    return L


def padded_fields(n, seed):
    phi, b = srt_fields.int_noise_fields(n, seed=seed, phi_log2=-33, b_log2=-37)
    pad = lambda f: np.ascontiguousarray(np.pad(f, ((1, 2), (1, 2), (1, 2)), mode="wrap"), np.float32)
    F = [pad(b[..., c]) for c in range(3)] + [pad(phi)]
    return F, (ctypes.c_void_p * 4)(*[f.ctypes.data for f in F])


@pytest.mark.parametrize("n,nside,steps", [((16, 16, 16), 2, 20), ((11, 14, 9), 3, 25), ((5, 3, 4), 1, 11),
                                           ((1, 2, 3), 1, 5)])
def test_layouts_trace_alike(host, n, nside, steps):
    F, ptrs = padded_fields(n, 7)
    count = 12 * nside * nside
    maps = np.zeros((6, count, 6), np.float32)
    flags = np.zeros((6, count), np.int32)
    host.layout_maps(ptrs, *n, nside, count, steps, maps.ctypes.data, flags.ctypes.data)
    assert np.all(np.isfinite(maps))
    for k in (1, 2, 4, 5):  # 0-2 second differences, 3-5 four taps
        assert np.array_equal(maps[k].view(np.uint32), maps[k // 3 * 3].view(np.uint32))
        assert np.array_equal(flags[k], flags[k // 3 * 3])


def diff2(a, ax):
    return np.roll(a, 1, ax) - 2 * a + np.roll(a, -1, ax)


@pytest.mark.parametrize("n,hot", [((12, 9, 14), 0), ((40, 36, 33), 1), ((40, 36, 33), 0)])
def test_cell_scatter_equals_tap_scatter(host, n, hot):
    """FP32 sums of the same products in another order: 1e-5 of the largest."""
    rng = np.random.default_rng(3)
    F, ptrs = padded_fields(n, 9)
    count = 300
    theta, phi = np.arccos(rng.uniform(-1, 1, count)), rng.uniform(0, 2 * np.pi, count)
    s = rng.uniform(0, 1.5 * max(n), count).astype(np.float32)
    d = (rng.standard_normal((count, 19)) * 1e-3).astype(np.float32)
    fb = rng.standard_normal(19).astype(np.float32)
    shape = (n[2] + 3, n[1] + 3, n[0] + 3)
    yb = np.zeros((3, count, 19), np.float32)
    rows = np.zeros((4,) + shape, np.float32)
    cells = np.zeros((4,) + shape + (4,), np.float32)
    side = host.hot_side()
    copies = np.zeros((4, side, side, side, 4), np.float32)
    host.layout_vjp(ptrs, *n, count, theta.ctypes.data, phi.ctypes.data, s.ctypes.data, d.ctypes.data,
                    fb.ctypes.data, yb.ctypes.data, rows.ctypes.data, cells.ctypes.data, copies.ctypes.data, hot)
    assert np.array_equal(yb[1].view(np.uint32), yb[0].view(np.uint32))
    assert np.array_equal(yb[2].view(np.uint32), yb[0].view(np.uint32))
    assert bool(np.any(copies)) == bool(hot)
    g = cells.astype(np.float64)
    if hot:
        lo = [m // 2 - side // 2 for m in n]
        g[:, lo[2]:lo[2] + side, lo[1]:lo[1] + side, lo[0]:lo[0] + side] += copies
    # nothing at the padded edges the transpose's neighbours would leave the grid from
    assert not np.any(g[:, :, [0, -1]]) and not np.any(g[:, :, :, [0, -1]])
    got = g[..., 0] + diff2(g[..., 1], 2) + diff2(g[..., 2], 3) + diff2(diff2(g[..., 3], 2), 3)
    for c in range(4):
        scale = np.abs(rows[c]).max()
        assert scale > 0 and np.abs(got[c] - rows[c]).max() <= 1e-5 * scale, c


@pytest.mark.parametrize("t", [(0.0, 0.0, 0.0), (0.25, 0.5, 0.875), (0.999999, 0.0, 0.5)])
def test_two_stages_scatter_as_one(host, t):
    """Two stages' cotangents added before they go to the cells: FP32 roundings of
    the same products, a few ulps of the largest (16 terms: 1e-6)."""
    n = (7, 6, 5)
    F, _ = padded_fields(n, 11)
    rng = np.random.default_rng(8)
    shape = (n[2] + 3, n[1] + 3, n[0] + 3, 4)
    for cell in ((0, 0, 0), (6, 5, 4), (3, 2, 1)):
        base = cell[0] + (n[0] + 3) * (cell[1] + (n[1] + 3) * cell[2])
        ta = np.array(t, np.float32)
        tb = np.clip(ta + np.float32(1e-5), 0, np.float32(1 - 2.0 ** -24)).astype(np.float32)
        qa, qb = rng.standard_normal((2, 10)).astype(np.float32)
        two, one = np.zeros(shape, np.float32), np.zeros(shape, np.float32)
        host.scatter_pair(F[0].ctypes.data, *n, base, *(a.ctypes.data for a in (ta, qa, tb, qb, two, one)))
        assert np.count_nonzero(one) > 0
        assert np.abs(two - one).max() <= 1e-6 * np.abs(one).max()
