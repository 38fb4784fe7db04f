"""A binary IVF that probes no list returns empty results, for results small enough to
be written straight into page-locked host memory and for larger ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,k", [(1, 1), (7, 10), (300, 10), (9000, 10)])
def test_no_probes_no_results(gn, nq, k):
    rng = np.random.default_rng(nq)
    db = rng.integers(0, 256, (5000, 32), dtype=np.uint8)
    ix = gn.IVFFlatBinaryIndex(nlist=16, nprobe=4)
    ix.set(db)
    before = ix.search_knn_arrays(db[:nq] if nq <= 5000 else np.resize(db, (nq, 32)), k)
    for nprobe in (0, -3):
        ix.set_nprobe(nprobe)
        q = np.resize(db, (nq, 32))
        idx, dist, cnt = ix.search_knn_arrays(q, k)
        assert (idx == -1).all() and (dist == 0).all() and (cnt == 0).all()
    ix.set_nprobe(4)
    after = ix.search_knn_arrays(np.resize(db, (nq, 32)), k)
    assert all(np.array_equal(a, b) for a, b in zip(before, after))
