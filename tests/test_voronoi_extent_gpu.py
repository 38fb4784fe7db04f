"""Rasters as wide and as high as the interface takes: the last pixels of the last tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [3, 40])
@pytest.mark.parametrize("wide", [True, False])
def test_largest_extent(gn, ns, wide):
    import torch
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    n = 2**31 - 1
    rng = np.random.default_rng(ns)
    seeds = rng.random((ns, 2), dtype=np.float32)
    long = torch.linspace(0, 1, n, device="cuda", dtype=torch.float32)
    short = torch.full((1,), 0.5, device="cuda", dtype=torch.float32)
    r = gn.voronoi_raster_device(torch.from_numpy(seeds).cuda(), long if wide else short, short if wide else long)
    ids = r.ids.view(-1)
    for at in (0, 1 << 30, n - 3000):
        v = long[at:at + 3000].cpu().numpy()
        along, across = (0, 1) if wide else (1, 0)
        a = v[:, None] - seeds[None, :, along]
        b = np.float32(0.5) - seeds[None, :, across]
        want = np.sqrt(a * a + b * b).argmin(1)
        assert np.array_equal(ids[at:at + 3000].cpu().numpy(), want)
    del r, ids, long
    torch.cuda.empty_cache()
