"""Tensor-core shortlist over fewer rows than a tile, below, at and above the shortlist's
length: nothing is lost on the way to the re-rank."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 16, 17, 33, 48, 49, 63, 64, 65, 100, 128, 129, 200, 255, 256, 257, 300])
@pytest.mark.parametrize("shortlist,precision", [(16, "bf16"), (32, "fp8"), (56, "bf16")])
def test_few_rows(gn, n, shortlist, precision):
    rng = np.random.default_rng(n + shortlist)
    db = rng.standard_normal((n, 40), dtype=np.float32)
    ix = gn.FlatL2TCIndex(shortlist=shortlist, precision=precision)
    ix.set(db)
    ex = gn.FlatL2Index()
    ex.set(db)
    for nq in (1, 129, 3000):
        q = rng.standard_normal((nq, 40), dtype=np.float32)
        k = min(16, n)
        idx, dist = ix.search_knn_arrays(q, k)
        ei, ed = ex.search_knn_arrays(q, k)
        if n <= shortlist:  # every row is re-ranked
            assert np.array_equal(idx, ei) and np.array_equal(dist.view(np.uint32), ed.view(np.uint32))
        else:
            assert (idx >= 0).all() and (np.diff(dist, axis=1) >= 0).all()
            near = min(k, shortlist // 4)  # far inside the shortlist
            assert (idx[:, :near] == ei[:, :near]).mean() >= (0.99 if precision == "fp8" else 1.0)
            assert (dist >= ed).all()
            same = idx == ei
            assert np.array_equal(dist[same], ed[same])
