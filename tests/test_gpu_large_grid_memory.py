"""A grid whose cells would take three to four tenths of the device keeps planes and half
cells (48 bytes a voxel), so that a gradient beside it has the memory it needs; its maps
are the ones of planes by the same passes, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_of_a_large_grid(srt, monkeypatch):
    torch = pytest.importorskip("torch")
    n = 1160
    srt.release_cached_memory()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    if not total // 10 * 3 < 64 * (n + 3) ** 3 <= total // 5 * 2 or free < 180e9:
        pytest.skip("another device memory size, or taken")
    g = torch.Generator("cuda").manual_seed(3)
    phi = torch.randn((n, n, n), device="cuda", generator=g).mul_(1e-6)
    b = torch.randn((n, n, n, 3), device="cuda", generator=g).mul_(1e-8)
    nside, steps = 24, 12
    with srt.Fields(phi, b) as f:
        assert f.nbytes == 16 * (n + 3) ** 3 + 32 * (n + 3) ** 2 * (n + 2)
        half, _ = f.forward(nside, steps)
    srt.release_cached_memory()
    monkeypatch.setenv("SRT_FIELDS_LAYOUT", "planes")
    with srt.Fields(phi, b) as f:
        planes, _ = f.forward(nside, steps)
    assert np.array_equal(half.view(np.uint32), planes.view(np.uint32))
    del phi, b
    torch.cuda.empty_cache()
    srt.release_cached_memory()
