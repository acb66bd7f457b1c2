"""Lists of flagged rays between four and 64 per SM are re-traced in FP64: their maps
are the FP64 form's bit for bit, and so the same whether a sky is traced whole or in
batches (whose lists are shorter)."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


def test_medium_lists_equal_fp64(srt):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, nside, steps = 96, 128, 96
    phi, b = srt_fields.gaussian_fields_np(n, seed=29)
    phi, b = phi * np.float32(200), b * np.float32(200)  # 0.7 % of the rays flagged
    with srt.Fields(phi, b) as f:
        m64, _ = f.forward(nside, steps, precision="fp64")
        mn, _ = f.forward(nside, steps, precision="mixed", refine=False)
        mr, st = f.forward(nside, steps, precision="mixed")
        assert 4 * sms < st.refined_rays <= 64 * sms, st.refined_rays
        changed = np.any(mr.view(np.uint32) != mn.view(np.uint32), axis=0)
        assert 4 * sms < changed.sum() <= st.refined_rays
        assert np.array_equal(mr[:, changed].view(np.uint32), m64[:, changed].view(np.uint32))
        for k in range(12):
            part, _ = f.forward(nside, steps, k * nside * nside, nside * nside, precision="mixed")
            whole = mr[:, k * nside * nside:(k + 1) * nside * nside]
            assert np.array_equal(part.view(np.uint32), whole.view(np.uint32))


def test_lists_longer_than_a_round_of_warps(srt, monkeypatch):
    """More flagged rays than the launch has warps (16 per SM): in FP64 bit for bit, in
    double-float (SRT_REFINE_DD_MIN=0) to four float ulps or 1e-6 of the map's rms, but
    for a few rays that pass a face within its rounding."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, nside, steps = 64, 640, 110
    phi, b = srt_fields.gaussian_fields_np(n, seed=6)
    with srt.Fields(phi * np.float32(50), b * np.float32(50)) as f:
        m64, _ = f.forward(nside, steps, precision="fp64")
        mn, _ = f.forward(nside, steps, refine=False)
        mr, st = f.forward(nside, steps)
        assert 16 * sms < st.refined_rays <= 64 * sms, st.refined_rays
        monkeypatch.setenv("SRT_REFINE_DD_MIN", "0")
        md, _ = f.forward(nside, steps)
    changed = np.any(mr.view(np.uint32) != mn.view(np.uint32), axis=0)
    assert np.array_equal(mr[:, changed].view(np.uint32), m64[:, changed].view(np.uint32))
    assert 16 * sms < changed.sum() <= st.refined_rays
    assert np.array_equal(md[:, ~changed].view(np.uint32), mn[:, ~changed].view(np.uint32))
    a, c = md[:, changed], m64[:, changed]
    ulps = np.abs(a.view(np.int32).astype(np.int64) - c.view(np.int32).astype(np.int64))
    rms = np.sqrt(np.mean((m64 - m64.mean(axis=1, keepdims=True)).astype(np.float64) ** 2, axis=1))
    off = (ulps > 4) & (np.abs(a - c) > 1e-6 * rms[:, None])
    assert np.mean(np.any(off, axis=0)) <= 2e-3
