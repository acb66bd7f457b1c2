"""The scratch pool keeps at most 8 GiB: after a gradient, a forward with a tape and
the tape's end, whose scratch is larger, the device has the rest back, with no
synchronisation by the caller."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu

KEEP = 8 << 30
SLACK = 256 << 20  # the pools' granularity, the context's own allocations


def test_scratch_above_the_bound_is_returned(srt):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("device memory is short")
    n, nside, steps = 48, 288, 64  # checkpoints every step: 65 x 152 B x 995,328 rays = 9.8 GB
    npix = 12 * nside * nside
    phi, b = srt_fields.gaussian_fields_np(n, seed=4)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dphi = torch.empty((n, n, n), device="cuda")
    w = torch.randn((6, npix), device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    out = torch.empty((6, npix), device="cuda")
    with srt.Fields(dev(phi), dev(b)) as f:
        f.forward(nside, 1, out=out)  # what a first call loads stays
        torch.cuda.synchronize()
        srt.release_cached_memory()
        free = torch.cuda.mem_get_info()[0]
        used = lambda: free - torch.cuda.mem_get_info()[0]
        for _ in range(2):
            f.vjp(nside, steps, w, dphi=dphi, wrt=("phi",), ckpt_every=1)
            assert used() <= KEEP + SLACK, used()
        _, tape, _ = f.forward_tape(nside, steps, ckpt_every=1, out=out)
        assert used() <= tape.nbytes + KEEP + SLACK, (used(), tape.nbytes)
        assert tape.nbytes > KEEP
        tape.vjp(w, dphi=dphi, wrt=("phi",))
        assert used() <= tape.nbytes + KEEP + SLACK, (used(), tape.nbytes)
        tape.close()
        assert used() <= KEEP + SLACK, used()
    srt.release_cached_memory()
