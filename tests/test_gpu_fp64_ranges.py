"""FP64 ranges on both sides of where five warps, one warp or one lane trace a ray give
the full sky's maps, bit for bit."""
import numpy as np
import pytest

import srt_fields

pytestmark = pytest.mark.gpu


def test_fp64_ranges_equal_the_sky(srt):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    phi, b = srt_fields.gaussian_fields_np((40, 37, 42), seed=5)
    nside, steps = 48, 12
    with srt.Fields(phi, b) as f:
        full, _ = f.forward(nside, steps, precision="fp64")
        for count in (1, 4 * sms, 4 * sms + 1, 140 * sms, 140 * sms + 1):
            part, _ = f.forward(nside, steps, 777, count, precision="fp64")
            assert np.array_equal(part.view(np.uint32), full[:, 777:777 + count].view(np.uint32)), count
