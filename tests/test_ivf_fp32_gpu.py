"""Edges of the FP32 IVF engine against the oracle: lists shorter and longer than
an item's rows, result counts around the buffers and the bound's sample, batches
planned by one block and by several, tied rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _index(gn, data, cent, labels, n_probe):
    ix = gn.IVFFlatL2Index(n_clusters=len(cent), n_probe=n_probe)
    ix.set_assigned(data, cent, labels)
    return ix


def _lattice(n, d, nlist, seed, biggest):
    """Rows on a small lattice (every inner product is exact in FP32, so the expanded
    form has no rounding to differ by), list 0 with `biggest` rows, the rest split at
    random; centroids apart along the first coordinate.  (One list or all of them are
    probed: distances to several centroids repeat.)"""
    rng = np.random.default_rng(seed)
    labels = np.r_[np.zeros(biggest, np.int32), rng.integers(1, nlist, n - biggest).astype(np.int32)]
    rng.shuffle(labels)
    cent = np.zeros((nlist, d), np.float32)
    cent[:, 0] = 8.0 * np.arange(nlist)
    data = cent[labels] + rng.integers(-3, 4, (n, d)).astype(np.float32)
    return data, cent, labels, rng


@pytest.mark.parametrize("n,d,nlist,biggest,nq,n_probe,k", [
    (300, 3, 4, 200, 1, 1, 5), (5000, 17, 40, 700, 65, 1, 10), (9000, 32, 20, 5000, 130, 20, 33),
    (20_000, 130, 250, 1500, 700, 250, 12), (4000, 600, 12, 900, 40, 12, 128), (8000, 40, 9, 4000, 33, 9, 129),
    (6000, 16, 30, 2500, 20, 30, 256), (1200, 8, 250, 3, 300, 1, 20), (30_000, 64, 2, 29_000, 100, 2, 10),
])
def test_equals_oracle_on_exact_arithmetic(gn, oracle, n, d, nlist, biggest, nq, n_probe, k):
    data, cent, labels, rng = _lattice(n, d, nlist, n + d, biggest)
    q = cent[rng.integers(0, nlist, nq)] + rng.integers(-3, 4, (nq, d)).astype(np.float32)
    q[: nq // 2] = cent[0] + rng.integers(-3, 4, (nq // 2, d)).astype(np.float32)
    ix = _index(gn, data, cent, labels, n_probe)
    idx, dist, cnt = ix.search_knn_arrays(q, k)
    oi, od, oc = oracle.ivfl2_search(data, cent, labels, q, k, n_probe)
    assert np.array_equal(cnt, oc)
    for i in range(nq):
        assert np.array_equal(dist[i, :cnt[i]], od[i, :cnt[i]])
        assert np.array_equal(idx[i, :cnt[i]], oi[i, :cnt[i]])


def test_identical_rows(gn):
    """One list of 3,000 equal rows: the k lowest rows, whatever fills the buffers."""
    data = np.ones((3000, 20), np.float32)
    ix = _index(gn, data, data[:1], np.zeros(3000, np.int32), 1)
    for k in (1, 40, 200):
        idx, dist, cnt = ix.search_knn_arrays(np.ones((70, 20), np.float32), k)
        assert (cnt == k).all() and (dist == 0).all() and (idx == np.arange(k)).all()
