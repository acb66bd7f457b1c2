"""A handle whose cells find no room keeps planes and half cells, or planes alone: the
same maps and gradients as from cells, bit for bit (SRT_FIELDS_LAYOUT takes the room
away). Full skies and the small ranges that four lanes share, odd extents, a grid
smaller than the copies around the observer, the forward / gradient pair and both
accumulations."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("n", [(44, 37, 40), (13, 9, 21)])
def test_layouts_agree(srt, monkeypatch, n):
    phi, b = srt_fields.gaussian_fields_np(n, seed=19)
    phi, b = phi * np.float32(30), b * np.float32(30)
    nside, steps = 24, 40  # 6,912 rays: a lane each; ranges of up to 4,864 four lanes
    rng = np.random.default_rng(2)
    ranges = [(begin, count, rng.standard_normal((6, count)).astype(np.float32))
              for begin, count in ((0, 12 * nside * nside), (1000, 900), (5, 1))]
    pvox = (n[0] + 3) * (n[1] + 3) * (n[2] + 3)
    pairs = (n[0] + 3) * (n[1] + 2) * (n[2] + 3)
    got = {}
    for layout, nbytes in (("cells", 64 * pvox), ("half", 16 * pvox + 32 * pairs), ("planes", 16 * pvox)):
        monkeypatch.setenv("SRT_FIELDS_LAYOUT", layout)
        out = got[layout] = []
        # extents are (n0, n1, n2), the arrays (n2, n1, n0)
        with srt.Fields(phi, b) as f:
            assert f.nbytes == nbytes
            for begin, count, w in ranges:
                m, st = f.forward(nside, steps, begin, count)
                maps, tape, _ = f.forward_tape(nside, steps, begin, count, ckpt_every=7)
                out += [m, np.float32([st.refined_rays]), maps]
                for det in (True, False):
                    out += list(f.vjp(nside, steps, w, begin, count, deterministic=det, ckpt_every=7)[:2])
                    out += list(tape.vjp(w, deterministic=det)[:2])
                tape.close()
    for layout in ("half", "planes"):
        for k, (a, c) in enumerate(zip(got[layout], got["cells"])):
            k %= 11
            if k < 3:
                assert np.array_equal(bits(a), bits(c)), (layout, k)
            else:
                # fixed point: the scalar FP32 expressions of two kernel variants may round
                # in another order (test_gpu_parity's bound); FP32 atomics: sums in another
                # order too (test_gpu_paired_scatter's)
                bound = 1e-6 if k < 7 else 1e-4
                assert np.abs(a - c).max() <= bound * np.abs(c).max(), (layout, k)
