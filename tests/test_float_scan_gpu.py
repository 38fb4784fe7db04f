"""Edges of the exact float scan against the oracle: batch sizes around its
queries-per-warp steps, result counts around its buffer sizes, row widths around
its boxes and remainders, row counts around its stages, ties, and values that are
not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INDEX = {"l2": "FlatL2Index", "l1": "FlatL1Index", "linf": "FlatChebyshevIndex"}


def _check(gn, oracle, metric, db, q, k):
    ix = getattr(gn, INDEX[metric])()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    oi, od = oracle.knn_float(metric, db, q, k)
    assert np.array_equal(idx, oi)
    assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("n,d,nq,k", [
    (1, 1, 1, 1), (33, 3, 2, 33), (129, 4, 3, 10), (257, 5, 4, 64), (1000, 7, 5, 65), (4099, 8, 8, 5),
    (4097, 12, 9, 97), (3001, 15, 16, 256), (2049, 31, 17, 200), (5003, 32, 33, 1), (6000, 33, 7, 32),
    (2000, 63, 40, 33), (3000, 64, 64, 64), (1999, 65, 70, 12), (1500, 97, 100, 100), (1003, 128, 130, 17),
    (700, 257, 19, 9), (300, 1030, 6, 21), (65_537, 16, 600, 3), (300_001, 10, 3, 150), (120, 9001, 2, 5),
])
def test_equals_oracle(gn, oracle, metric, n, d, nq, k):
    rng = np.random.default_rng(n + d)
    _check(gn, oracle, metric, rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32), k)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("k", [3, 40, 180])
def test_ties_go_to_the_lower_index(gn, oracle, metric, k):
    """Coordinates of few values: most rows are at distances that repeat."""
    rng = np.random.default_rng(k)
    db = rng.integers(0, 3, (9000, 6)).astype(np.float32)
    _check(gn, oracle, metric, db, db[rng.integers(0, 9000, 37)], k)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
def test_rows_in_descending_distance(gn, oracle, metric):
    """Every row is nearer than all before it: buffers fill and are cut throughout."""
    n = 20_000
    db = np.linspace(2.0, 0.0, n, dtype=np.float32)[:, None] * np.ones((1, 9), np.float32)
    for k in (1, 20, 100):
        _check(gn, oracle, metric, db, np.zeros((6, 9), np.float32), k)


def test_rows_that_are_not_finite(gn):
    """Infinite distances come after the finite ones, in row order; more results
    than finite rows are asked for."""
    rng = np.random.default_rng(4)
    db = rng.random((500, 8), dtype=np.float32)
    db[100:400] = np.inf
    q = rng.random((5, 8), dtype=np.float32)
    for name in INDEX.values():
        ix = getattr(gn, name)()
        ix.set(db)
        idx, dist = ix.search_knn_arrays(q, 250)
        assert np.isfinite(dist[:, :200]).all() and np.isposinf(dist[:, 200:]).all()
        assert (idx[:, 200:] == np.arange(100, 150)).all()
