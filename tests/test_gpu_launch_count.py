"""srt_stats.kernels of a gradient from a tape (every segment recomputed): the
cotangent kernel, per segment the recompute and the sweep, the merges of the copies
around the observer (FP32) and the folds."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside", [4, 32])  # four lanes per ray, and one
@pytest.mark.parametrize("det", [False, True])
def test_launches_of_a_tape_gradient(srt, nside, det):
    phi, b = srt_fields.gaussian_fields_np(40, seed=3)
    w = np.ones((6, 12 * nside * nside), np.float32)
    with srt.Fields(phi, b) as f:
        _, tape, _ = f.forward_tape(nside, 20, ckpt_every=6)  # 4 segments
        _, _, st = tape.vjp(w, deterministic=det)
        tape.close()
    assert st.kernels == 1 + 4 * 2 + (0 if det else 4) + 4
