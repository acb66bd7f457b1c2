"""Grids the MIXED form traces by its four-tap passes (planes from 512^3 on with
SRT_FIELDS_NO_PAIRS; planes or row pairs where cells would not fit the device):
against the FP64 form, small ranges (four lanes per ray) against the full sky bit
for bit, the tape's maps against the forward's, and gradients against the default
handle's."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import srt_fields
from conftest import map_errors

pytestmark = pytest.mark.gpu

# test_gpu_parity's bounds on MIXED against the FP64 form
RMS, MAX = 1e-5, 1e-4


def check_handle(f, nside, steps, label):
    npix = 12 * nside * nside
    full, st = f.forward(nside, steps, precision="mixed")
    want, _ = f.forward(nside, steps, precision="fp64")
    for m, (rms, mx) in enumerate(map_errors(full, want)):
        assert rms <= RMS and mx <= MAX, (label, m, rms, mx)
    # one ray, a few, a warp and one more of eight-ray groups, a RING range off any edge
    for begin, count in ((0, 1), (npix // 2 + 3, 7), (npix - 33, 33), (npix // 3, 1000)):
        part, _ = f.forward(nside, steps, begin, count, precision="mixed")
        assert np.array_equal(part.view(np.uint32), full[:, begin:begin + count].view(np.uint32)), (label, begin)
    return full, st


def test_planes_of_a_large_grid(srt):
    torch = pytest.importorskip("torch")
    phi, b = srt_fields.gaussian_fields_torch(512, seed=21)
    nside, steps = 48, 40
    npix = 12 * nside * nside
    with srt.Fields(phi, b, pairs=False) as f:
        assert f.nbytes == 16 * 515 ** 3
        full, _ = check_handle(f, nside, steps, "planes 512^3")
        maps, tape, _ = f.forward_tape(nside, steps, ckpt_every=7)
        assert np.array_equal(maps.view(np.uint32), full.view(np.uint32))
        w = torch.randn((6, npix), device="cuda", generator=torch.Generator("cuda").manual_seed(5))
        g4 = torch.empty_like(phi)
        gt = torch.empty_like(phi)
        f.vjp(nside, steps, w, precision="mixed", dphi=g4, deterministic=True, wrt=("phi",))
        tape.vjp(w, dphi=gt, deterministic=True, wrt=("phi",))
        assert torch.equal(g4, gt)  # any checkpoint interval, from the tape or not
        tape.close()
    with srt.Fields(phi, b) as f:
        g = torch.empty_like(phi)
        f.vjp(nside, steps, w, precision="mixed", dphi=g, deterministic=True, wrt=("phi",))
    # FP32 trajectories of two roundings: 1e-7 relative in each stage's taps, 160
    # stages, sums of both signs over a voxel's rays
    assert float((g4 - g).abs().max()) <= 2e-5 * float(g.abs().max())


def test_planes_and_row_pairs_where_cells_would_not_fit(srt):
    torch = pytest.importorskip("torch")
    n = 1260
    free, total = torch.cuda.mem_get_info()
    if 64 * (n + 3) ** 3 <= total // 5 * 2 or free < 160e9:
        pytest.skip("another device memory size, or taken")
    g = torch.Generator("cuda").manual_seed(3)
    phi = torch.randn((n, n, n), device="cuda", generator=g).mul_(1e-6)
    b = torch.randn((n, n, n, 3), device="cuda", generator=g).mul_(1e-8)
    nside, steps = 24, 12
    maps = {}
    for pairs in (True, False):
        with srt.Fields(phi, b, pairs=pairs) as f:
            planes = 16 * (n + 3) ** 3
            assert f.nbytes == planes + (32 * (n + 3) ** 2 * (n + 2) if pairs else 0)
            maps[pairs], _ = check_handle(f, nside, steps, "row pairs" if pairs else "planes")
    assert np.array_equal(maps[True].view(np.uint32), maps[False].view(np.uint32))
    del phi, b
    torch.cuda.empty_cache()
    srt.release_cached_memory()
