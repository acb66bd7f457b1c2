"""A grid too large for cells on any handle (SRT_FIELDS_LAYOUT=pairs makes a small one
such): the four taps from row pairs and from planes give the same maps, bit for bit, and
the same gradients; both against the second differences of a default handle."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(44, 37, 40), (13, 9, 21)])
def test_row_pairs_equal_planes(srt, monkeypatch, n):
    phi, b = srt_fields.gaussian_fields_np(n, seed=19)
    nside, steps = 24, 40  # 6,912 rays: a lane each; ranges of up to 4,864 four lanes
    rng = np.random.default_rng(2)
    ranges = [(begin, count, rng.standard_normal((6, count)).astype(np.float32))
              for begin, count in ((0, 12 * nside * nside), (1000, 900), (5, 1))]
    pvox = (n[0] + 3) * (n[1] + 3) * (n[2] + 3)
    pairs = (n[0] + 3) * (n[1] + 2) * (n[2] + 3)
    got = {}
    for layout, nbytes in (("cells", 64 * pvox), ("pairs", 16 * pvox + 32 * pairs), ("planes", 16 * pvox)):
        if layout != "cells":
            monkeypatch.setenv("SRT_FIELDS_LAYOUT", "pairs")
        out = got[layout] = []
        with srt.Fields(phi, b, pairs=layout != "planes") as f:
            assert f.nbytes == nbytes
            for begin, count, w in ranges:
                m, st = f.forward(nside, steps, begin, count)
                maps, tape, _ = f.forward_tape(nside, steps, begin, count, ckpt_every=7)
                assert np.array_equal(m.view(np.uint32), maps.view(np.uint32))
                out.append(m)
                for det in (True, False):
                    out += list(f.vjp(nside, steps, w, begin, count, deterministic=det, ckpt_every=7)[:2])
                    out += list(tape.vjp(w, deterministic=det)[:2])
                tape.close()
    for k, (p, q, c) in enumerate(zip(got["pairs"], got["planes"], got["cells"])):
        k %= 9
        if k == 0:
            assert np.array_equal(p.view(np.uint32), q.view(np.uint32))
            # FP32 roundings of 160 stages: 1e-5 of each map's largest value
            assert np.all(np.abs(p - c).max(axis=1) <= 1e-5 * np.abs(c).max(axis=1) + 1e-12)
        else:
            # as in test_gpu_field_layouts; and against the other passes' trajectory, FP32
            # roundings of 160 stages summed over rays (test_gpu_four_taps: 2e-5)
            bound = 1e-6 if k < 5 else 1e-4
            assert np.abs(p - q).max() <= bound * np.abs(q).max(), k
            assert np.abs(p - c).max() <= 1e-4 * np.abs(c).max(), k
