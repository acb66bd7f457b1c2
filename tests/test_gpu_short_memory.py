"""A gradient whose larger scratch finds no room takes less of it instead of failing:
one segment's tape where several do not fit, and half the rays at a time. The allocation is made to fail on the host
(srt_debug_fail_alloc); the gradient keeps its bits (SRT_DETERMINISTIC)."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


def completes_without_failure_at(srt, call, allocations):
    """The results of the calls that completed although one of their allocations
    failed, by its index."""
    L = srt.lib()
    out = {}
    for after in range(allocations):
        L.srt_debug_fail_alloc(after)
        try:
            out[after] = call()
        except srt.SrtError as e:
            assert e.code == -3, str(e)
        finally:
            pending = L.srt_debug_fail_alloc(-1)
        assert pending == 0
    return out


@pytest.mark.parametrize("nside,precision,less", [(4, "mixed", 1), (32, "mixed", 5), (20, "fp64", 2)])
def test_gradient_with_less_scratch(srt, nside, precision, less):
    phi, b = srt_fields.gaussian_fields_np(24, seed=6)
    w = np.random.default_rng(7).standard_normal((6, 12 * nside * nside)).astype(np.float32)
    with srt.Fields(phi, b) as f:
        # 7 segments, all kept
        call = lambda: f.vjp(nside, 20, w, ckpt_every=3, deterministic=True, precision=precision)[:2]
        want = call()
        # outputs 2, ray list 3, weights 1, accumulators 4, range flag; then what goes by
        # rays: checkpoints, marks, bases, cotangents, segment records (FP64: the first
        # and the last; 192 rays: only the records of several segments)
        done = completes_without_failure_at(srt, call, 16)
        assert len([k for k in done if k >= 11]) >= less and all(k >= 11 for k in done), sorted(done)
        for g in done.values():
            for a, c in zip(g, want):
                assert np.array_equal(a.view(np.uint32), c.view(np.uint32))


def test_ref16_without_its_phi_plane(srt):
    """The phi plane that REF16 makes beside cells is only faster: without room for it the
    maps are the same."""
    phi, b = srt_fields.gaussian_fields_np((24, 21, 26), seed=6)
    with srt.Fields(phi, b) as f:
        assert f.nbytes == 64 * 27 * 24 * 29
        want, _ = f.forward(4, 16, precision="ref16")
    L = srt.lib()
    with srt.Fields(phi, b) as f:
        L.srt_debug_fail_alloc(3)  # after the three B planes
        try:
            got, _ = f.forward(4, 16, precision="ref16")
        finally:
            L.srt_debug_fail_alloc(-1)
        again, _ = f.forward(4, 16, precision="ref16")
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(again.view(np.uint32), want.view(np.uint32))
