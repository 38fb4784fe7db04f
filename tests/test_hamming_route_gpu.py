"""Hamming searches on both sides of the rules that choose between ordered lists and
appended candidates: few rows, rows of few bits (ties everywhere), and more than 64
results with many pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nbytes,nq,k", [
    (1, 8, 300, 1), (16, 33, 500, 8), (17, 33, 500, 8), (16, 8, 40, 9), (512, 64, 6000, 4), (513, 64, 6000, 4),
    (512, 64, 5999, 4), (300, 5, 7000, 8), (300, 5, 7000, 9), (511, 1, 24, 3), (512, 1, 24, 3), (512, 1, 23, 3),
    (15_000, 1, 90, 4), (15_000, 1, 9000, 1), (15_000, 1, 3000, 16), (15_000, 1, 3000, 17), (140_000, 2, 30, 8),
    (100_000, 115, 4139, 65), (100_000, 115, 4137, 65), (300_000, 64, 2100, 128), (100_000, 100, 1000, 129),
    (20_000, 16, 9000, 1), (20_000, 16, 9000, 15),
])
def test_equals_oracle(gn, oracle, n, nbytes, nq, k):
    rng = np.random.default_rng(n + nbytes + k)
    db = rng.integers(0, 256, (n, nbytes), dtype=np.uint8)
    q = rng.integers(0, 256, (nq, nbytes), dtype=np.uint8)
    ix = gn.FlatHammingIndex()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    for s in (slice(0, 40), slice(max(0, nq - 40), nq)):
        oi, od = oracle.knn_hamming(db, q[s], k)
        assert np.array_equal(idx[s], oi) and np.array_equal(dist[s], od)
