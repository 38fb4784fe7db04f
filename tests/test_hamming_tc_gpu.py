"""Large Hamming batches (answered on the tensor cores) against the oracle: every
width class of a row, result counts up to the largest, ragged batches, tied and
repeated rows, and searches after a new set()."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, nb, nq, seed, distinct=None):
    rng = np.random.default_rng(seed)
    db = rng.integers(0, 256, (distinct or n, nb), dtype=np.uint8)
    if distinct:
        db = db[rng.integers(0, distinct, n)]
    q = db[rng.integers(0, n, nq)].copy()
    q[:, 0] ^= rng.integers(0, 256, nq, dtype=np.uint8)
    return db, q


@pytest.mark.parametrize("n,nb,nq,k", [
    (32_768, 64, 4096, 10),    # the smallest table, whole tiles of rows and queries
    (33_001, 64, 4001, 1),     # a ragged last tile and batch
    (40_011, 33, 6001, 33), (60_000, 16, 8500, 64), (70_001, 8, 14_501, 7),
    (50_000, 20, 8300, 5), (45_000, 96, 2000, 10), (33_333, 128, 2100, 3), (32_800, 500, 600, 10),
    (200_000, 64, 700, 40),
    (600_000, 64, 257, 10),    # few queries over many chunks
])
def test_equals_oracle(gn, oracle, n, nb, nq, k):
    db, q = _data(n, nb, nq, seed=n + nb)
    ix = gn.FlatHammingIndex()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    oi, od = oracle.knn_hamming(db, q, k)
    assert np.array_equal(idx, oi) and np.array_equal(dist, od)


def test_repeated_rows_tie_to_the_lower_index(gn, oracle):
    """500 distinct rows 80 times each: more rows at every distance than results,
    so the answer is decided by row order alone."""
    db, q = _data(40_000, 64, 3300, seed=3, distinct=500)
    ix = gn.FlatHammingIndex()
    ix.set(db)
    for k in (10, 64):
        idx, dist = ix.search_knn_arrays(q, k)
        oi, od = oracle.knn_hamming(db, q, k)
        assert np.array_equal(idx, oi) and np.array_equal(dist, od)


def test_new_rows_replace_the_old_ones(gn, oracle):
    ix = gn.FlatHammingIndex()
    for seed, n, nb in ((5, 40_000, 64), (6, 50_000, 64), (7, 40_000, 32)):
        db, q = _data(n, nb, 6500, seed)
        ix.set(db)
        idx, dist = ix.search_knn_arrays(q, 10)
        oi, od = oracle.knn_hamming(db, q, 10)
        assert np.array_equal(idx, oi) and np.array_equal(dist, od)
