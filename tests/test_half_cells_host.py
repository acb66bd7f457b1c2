"""The MIXED form on half cells (value and second difference along y), built for the
host: the maps, guard flags and state cotangents of planes, bit for bit. Odd, non-cubic
and very small grids, rays that wrap around the box."""
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
    out = str(tmp_path_factory.mktemp("half") / "libhalf.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + os.path.join(ROOT, "snapshot-raytracer_gb300", "csrc"), "-I" + cuda_inc,
                        os.path.join(ROOT, "tests", "half_shim.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    L = ctypes.CDLL(out)
    P, I, Q = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    L.half_compare.argtypes = [P, I, I, I, Q, Q, I, ctypes.c_float, P, P, P, P, P]
    return L


@pytest.mark.parametrize("n,nside,steps", [((16, 16, 16), 2, 20), ((11, 14, 9), 3, 25), ((5, 3, 4), 1, 11),
                                           ((1, 2, 3), 1, 5), ((3, 1, 2), 1, 5)])
def test_half_cells_equal_planes(host, n, nside, steps):
    phi, b = srt_fields.int_noise_fields(n, seed=7, phi_log2=-33, b_log2=-37)
    pad = lambda f: np.ascontiguousarray(np.pad(f, ((1, 2), (1, 2), (1, 2)), mode="wrap"), np.float32)
    F = [pad(b[..., c]) for c in range(3)] + [pad(phi)]
    count = 12 * nside * nside
    rng = np.random.default_rng(1)
    d = (1e-3 * rng.standard_normal(19)).astype(np.float32)
    fb = rng.standard_normal(19).astype(np.float32)
    maps, flags = np.zeros((2, count, 6), np.float32), np.zeros((2, count), np.int32)
    yb = np.zeros((2, count, 19), np.float32)
    host.half_compare((ctypes.c_void_p * 4)(*[f.ctypes.data for f in F]), *n, nside, count, steps, 7.3, d.ctypes.data,
                      fb.ctypes.data, maps.ctypes.data, flags.ctypes.data, yb.ctypes.data)
    assert np.all(np.isfinite(maps)) and np.all(np.isfinite(yb)) and np.any(yb)
    assert np.array_equal(maps[0].view(np.uint32), maps[1].view(np.uint32))
    assert np.array_equal(flags[0], flags[1])
    assert np.array_equal(yb[0].view(np.uint32), yb[1].view(np.uint32))
