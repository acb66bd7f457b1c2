"""SRT_FIELDS_NO_PAIRS from 80^3 voxels on takes the four taps: odd extents against the
FP64 form, small ranges against the full sky and the pair's maps bit for bit, and a sky
that fills the device no slower than by the second differences formed on the spot."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import srt_fields
from test_gpu_four_taps import check_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(79, 79, 79), (80, 80, 82), (165, 97, 61)])  # below and above 2^19
def test_planes_against_fp64(srt, n):
    phi, b = srt_fields.gaussian_fields_np(n, seed=8)
    nside, steps = 30, 50
    with srt.Fields(phi, b, pairs=False) as f:
        full, _ = check_handle(f, nside, steps, "planes")
        maps, tape, _ = f.forward_tape(nside, steps, ckpt_every=9)
        tape.close()
        assert np.array_equal(maps.view(np.uint32), full.view(np.uint32))


def test_planes_are_not_slower_than_second_differences(srt, monkeypatch):
    torch = pytest.importorskip("torch")
    phi, b = srt_fields.gaussian_fields_torch(256, seed=11)
    nside, steps = 128, 128
    out = torch.empty((6, 12 * nside * nside), device="cuda")

    def best(f):
        return min(f.forward(nside, steps, out=out, refine=False)[1].trace_ms for _ in range(6))

    with srt.Fields(phi, b, pairs=False) as f:
        flagged = best(f)
    monkeypatch.setenv("SRT_FIELDS_LAYOUT", "planes")  # second differences from planes
    with srt.Fields(phi, b) as f:
        spot = best(f)
    assert flagged <= 0.96 * spot, (flagged, spot)  # 11.1 against 12.1 ms


@pytest.mark.parametrize("rays", [768, 3072])
def test_small_ranges_of_planes(srt, monkeypatch, rays):
    """Ranges that four lanes share: no slower either (128^3, 48 steps, 3,072 rays: 0.260
    against 0.300 ms)."""
    torch = pytest.importorskip("torch")
    phi, b = srt_fields.gaussian_fields_torch(128, seed=11)
    out = torch.empty((6, rays), device="cuda")
    nside = int((rays / 12) ** 0.5)

    def best(f):
        return min(f.forward(nside, 48, out=out, refine=False)[1].trace_ms for _ in range(10))

    with srt.Fields(phi, b, pairs=False) as f:
        flagged = best(f)
    monkeypatch.setenv("SRT_FIELDS_LAYOUT", "planes")
    with srt.Fields(phi, b) as f:
        spot = best(f)
    assert flagged <= spot, (flagged, spot)
