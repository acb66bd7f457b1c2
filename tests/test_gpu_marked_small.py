"""Rays marked near a cell face in ranges that four lanes share: the recompute of a
segment takes them with the others, by the four taps. Any checkpoint interval, with and
without a tape, gives the gradient's bits (SRT_DETERMINISTIC), and a range split so that
a lane traces each ray the same to FP32 sums."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(64, 64, 64), (45, 50, 39)])
def test_marked_rays_of_small_ranges(srt, n):
    phi, b = srt_fields.gaussian_fields_np(n, seed=6)
    phi, b = phi * np.float32(50), b * np.float32(50)  # no caustics: every gradient finite
    nside, steps = 32, 120  # 12,288 rays by a lane each; thirds by four
    npix = 12 * nside * nside
    w = np.random.default_rng(3).standard_normal((6, npix)).astype(np.float32) * np.float32(2.0 ** -14)
    with srt.Fields(phi, b) as f:
        whole = f.vjp(nside, steps, w, deterministic=True, ckpt_every=7)[:2]
        summed = [np.zeros_like(g) for g in whole]
        marked = 0
        for k in range(3):
            lo, cnt = k * npix // 3, npix // 3
            wk = np.ascontiguousarray(w[:, lo:lo + cnt])
            _, tape, st = f.forward_tape(nside, steps, lo, cnt, ckpt_every=11)
            marked += st.refined_rays
            got = tape.vjp(wk, deterministic=True)[:2]
            tape.close()
            for ck in (1, 5, 120):  # all segments kept, some kept, one
                other = f.vjp(nside, steps, wk, lo, cnt, deterministic=True, ckpt_every=ck)[:2]
                for a, c in zip(got, other):
                    assert np.array_equal(a.view(np.uint32), c.view(np.uint32)), (k, ck)
            for s, v in zip(summed, got):
                s += v
    assert marked > 3
    for g, s in zip(whole, summed):
        # one float ulp per kernel variant, FP32 sums of the parts: 2e-6 of the largest
        assert np.abs(g - s).max() <= 2e-6 * np.abs(g).max()
