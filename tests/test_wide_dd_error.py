"""The double-float warp-per-ray trace's own error, its lanes emulated on the host
(wide_shim.cpp), against the one-lane FP64 form: no larger than that of plain
double-word sums for the state (one lane, 48^3, 60 steps: median position error
2.9e-13 grid units, dA 2.8e-13). 192 rays, so the median is good to ~10 %; an update
that carries y's sum through a compensated chain gives 4.1e-13 and 4.2e-13."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import srt_fields
from test_wide_host import host  # noqa: F401  (the fixture)


def test_double_float_error(host):  # noqa: F811
    n, nside, steps = 48, 4, 60
    phi, b = srt_fields.gaussian_fields_np(n, seed=3)
    pad = lambda f: np.ascontiguousarray(np.pad(f, ((1, 2), (1, 2), (1, 2)), mode="wrap"), np.float32)
    F = [pad(phi)] + [pad(b[..., c]) for c in range(3)]
    count = 12 * nside * nside
    y = [np.zeros((count, 19)) for _ in range(4)]
    host.trace_states(*[f.ctypes.data for f in F], n, n, n, nside, 0, count, steps, *[v.ctypes.data for v in y])
    err = np.abs(y[2] - y[0])
    assert np.median(err[:, :3].max(axis=1)) <= 3.4e-13
    assert np.median(err[:, 12]) <= 3.4e-13
