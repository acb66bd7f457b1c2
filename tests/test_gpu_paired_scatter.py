"""The FP32 sweep adds two stages' tap cotangents before they go to memory. Fields
strong enough that the two often lie in different cells; each gradient against the
fixed-point one, which scatters every stage by itself, over odd and even segment
lengths (a segment's first and last stages have no partner)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [True, False], ids=["cells", "planes"])
@pytest.mark.parametrize("ckpt", [1, 2, 5, 16])
def test_paired_scatter_equals_single(srt, pairs, ckpt):
    rng = np.random.default_rng(31)
    n, nside, steps = 40, 24, 16  # more rays than the four-lane sweep takes
    phi = (1e-3 * rng.standard_normal((n, n, n))).astype(np.float32)
    b = (1e-3 * rng.standard_normal((n, n, n, 3))).astype(np.float32)
    w = rng.standard_normal((6, 12 * nside * nside)).astype(np.float32)
    with srt.Fields(phi, b, pairs=pairs) as f:
        want = f.vjp(nside, steps, w, precision="mixed", ckpt_every=ckpt, deterministic=True)
        for wrt in (("phi", "b"), ("phi",), ("b",)):
            got = f.vjp(nside, steps, w, precision="mixed", ckpt_every=ckpt, wrt=wrt)
            for name, g, d in (("phi", got[0], want[0]), ("b", got[1], want[1])):
                if name not in wrt:
                    assert g is None
                    continue
                # FP32 sums of up to ~1e4 terms of both signs in a voxel, each good to
                # ~1e-6: 1e-4 of the largest entry; a stage lost or counted twice is 1e-2
                assert np.abs(g - d).max() <= 1e-4 * np.abs(d).max(), (wrt, name)
