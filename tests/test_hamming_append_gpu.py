"""Appended-candidate Hamming scan against the oracle: one to eight queries a group, odd
words, buffers on both sides of 64 neighbours, ties, rows around a block's step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nbytes,nq,k", [
    (1, 1, 1, 1), (5, 16, 1, 9), (511, 17, 1, 10), (513, 32, 1, 256), (100_003, 64, 1, 10), (257, 33, 2, 64),
    (70_001, 48, 2, 65), (256, 8, 3, 32), (4099, 128, 4, 100), (30_000, 20, 5, 10), (30_000, 64, 9, 64),
    (20_000, 64, 33, 65), (129, 61, 70, 129), (3000, 4, 100, 200), (1000, 3000, 6, 20), (40_000, 16, 127, 1),
])
def test_hamming_equals_the_oracle(gn, oracle, n, nbytes, nq, k):
    rng = np.random.default_rng(n + nbytes + nq)
    db = rng.integers(0, 256, (n, nbytes), dtype=np.uint8)
    db[n // 2 :] = db[: n - n // 2]  # every distance twice: the lower index first
    q = rng.integers(0, 256, (nq, nbytes), dtype=np.uint8)
    q[0] = db[n // 3]
    ix = gn.FlatHammingIndex()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    oi, od = oracle.knn_hamming(db, q, min(k, n))
    assert np.array_equal(idx, oi) and np.array_equal(dist, od)
