"""The warp-per-ray and block-per-ray traces (srt_wide.cuh: the re-trace of
flagged rays and the FP64 form of small ranges), their lanes emulated on the
host: in FP64 they must
give the one-lane FP64 form's state bit for bit (all write the same fused
chains), in double-float the same state to ~1e-12. Odd, non-cubic and very
small grids, rays that wrap around the box, and the dA > 1/2 branch (off in
the first step, on after it)."""
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
    out = str(tmp_path_factory.mktemp("wide") / "libwide.so")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                        "-I" + os.path.join(ROOT, "snapshot-raytracer_gb300", "csrc"), "-I" + cuda_inc,
                        os.path.join(ROOT, "tests", "wide_shim.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    L = ctypes.CDLL(out)
    P, I, Q = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    L.trace_states.argtypes = [P, P, P, P, I, I, I, Q, Q, Q, I, P, P, P, P]
    return L


@pytest.mark.parametrize("n,nside,steps", [((16, 16, 16), 2, 12), ((11, 14, 9), 3, 17), ((5, 3, 4), 1, 9),
                                           ((1, 2, 3), 1, 4), ((24, 24, 24), 2, 1)])
def test_wide_equals_one_lane(host, n, nside, steps):
    phi, b = srt_fields.int_noise_fields(n, seed=5, phi_log2=-31, b_log2=-35)  # strong fields: every term counts
    pad = lambda f: np.ascontiguousarray(np.pad(f, ((1, 2), (1, 2), (1, 2)), mode="wrap"), np.float32)
    F = [pad(phi)] + [pad(b[..., c]) for c in range(3)]
    count = 12 * nside * nside
    y = [np.zeros((count, 19)) for _ in range(4)]
    host.trace_states(*[f.ctypes.data for f in F], *n, nside, 0, count, steps, *[v.ctypes.data for v in y])
    one, wide, ddf, block = y
    assert np.array_equal(one, wide) and np.array_equal(one, block)
    assert np.all(np.isfinite(one)) and (steps == 1 or np.abs(one[:, 16:18]).max() > 1e-6)
    # double-float: 2^-45 or so per operation, a few hundred operations deep, on O(1)..O(n) values; a ray
    # whose stage position lies within that of a cell face may take the other cell
    err = np.abs(ddf - one).max(axis=1) / np.abs(one).max(axis=1)
    assert np.median(err) <= 1e-12 and np.mean(err <= 1e-10) >= 0.9, np.sort(err)[-5:]
