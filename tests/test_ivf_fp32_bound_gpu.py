"""The FP32 IVF scan with and without its bound: batches, result counts and rows per
query on both sides of the rule that takes it, one index through batches that grow and
shrink its scratch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(n, d, nlist, seed):
    """Rows on a small lattice around far centroids: every product exact in FP32."""
    rng = np.random.default_rng(seed)
    labels = rng.integers(0, nlist, n).astype(np.int32)
    cent = np.zeros((nlist, d), np.float32)
    cent[:, 0] = 8.0 * np.arange(nlist)
    return cent[labels] + rng.integers(-3, 4, (n, d)).astype(np.float32), cent, labels, rng


@pytest.mark.parametrize("n,d,nlist", [(3000, 32, 6), (3000, 33, 6), (1500, 100, 3), (1700, 100, 3), (4000, 200, 2),
                                       (40_000, 300, 2)])
def test_equals_oracle(gn, oracle, n, d, nlist):
    data, cent, labels, rng = _lattice(n, d, nlist, n + d)
    ix = gn.IVFFlatL2Index(n_clusters=nlist, n_probe=nlist)
    ix.set_assigned(data, cent, labels)
    for nq in (1, 3, 4, 300, 5):
        q = cent[rng.integers(0, nlist, nq)] + rng.integers(-3, 4, (nq, d)).astype(np.float32)
        for k in (1, 32, 33, 128, 129):
            idx, dist, cnt = ix.search_knn_arrays(q, k)
            m = min(nq, 20)
            oi, od, oc = oracle.ivfl2_search(data, cent, labels, q[:m], k, nlist)
            assert np.array_equal(cnt[:m], oc)
            for i in range(m):
                assert np.array_equal(idx[i, :cnt[i]], oi[i, :cnt[i]]) and np.array_equal(dist[i, :cnt[i]], od[i, :cnt[i]])
