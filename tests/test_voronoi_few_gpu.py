"""Rasters of few seeds (every seed for every pixel) and of just more (by tiles), over
widths and heights at the edges of both, with ties and coordinates that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 5), (4, 8), (127, 9), (128, 16), (130, 1), (257, 700), (1100, 301),
                                 (2048, 2049)])
@pytest.mark.parametrize("ns", [1, 2, 8, 9, 10, 16, 17])
def test_few_seeds(gn, oracle, w, h, ns):
    import torch
    rng = np.random.default_rng(w * h + ns)
    seeds = rng.random((ns, 2), dtype=np.float32)
    if ns > 2:
        seeds[ns // 2] = seeds[0]  # a tie everywhere
    xs, ys = rng.random(w, dtype=np.float32), np.linspace(0, 1, h, dtype=np.float32)
    if w > 100:
        xs[7], xs[9] = np.nan, np.inf
    pal = rng.integers(0, 256, (3, 4), dtype=np.uint8)
    r = gn.voronoi_raster_device(torch.from_numpy(seeds).cuda(), torch.from_numpy(xs).cuda(),
                                 torch.from_numpy(ys).cuda(), palette=torch.from_numpy(pal).cuda(),
                                 with_distance=True)
    ids, dist = r.ids.cpu().numpy(), r.dist.cpu().numpy()
    rgba = r.rgba.cpu().numpy()
    dx = xs[None, :, None] - seeds[None, None, :, 0]
    dy = ys[:, None, None] - seeds[None, None, :, 1]
    with np.errstate(invalid="ignore", over="ignore"):
        d = np.sqrt(dx * dx + dy * dy)
    d = np.where(np.isnan(d), np.float32(np.inf), d)
    want = d.argmin(2)  # the first of equal distances
    assert np.array_equal(ids, want)
    assert np.array_equal(dist, np.take_along_axis(d, want[..., None], 2)[..., 0])
    assert np.array_equal(rgba, pal[want % 3])
