"""Large exact L2 batches (candidates from the tensor cores) against the oracle:
indices and distance bits equal for every layout of the split rows, for data that
the bound cannot separate (the FP32 scan answers then), for ties and for values
that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(gn, oracle, db, q, k, sub=None):
    ix = gn.FlatL2Index()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    again = ix.search_knn_arrays(q, k)  # the index may have gone over to the FP32 scan
    assert np.array_equal(idx, again[0]) and np.array_equal(dist.view(np.uint32), again[1].view(np.uint32))
    s = slice(None) if sub is None else slice(0, sub)
    oi, od = oracle.knn_float("l2", db, q[s], k)
    assert np.array_equal(idx[s], oi)
    assert np.array_equal(dist[s].view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("n,d,nq,k", [
    (32_768, 32, 1500, 5), (40_001, 31, 1300, 1), (50_000, 33, 1000, 32), (100_000, 32, 500, 10),
    (33_000, 128, 400, 10), (40_000, 100, 401, 7), (200_000, 128, 64, 20), (60_000, 21, 1251, 3),
    (33_333, 300, 160, 12), (32_800, 700, 70, 4),
])
def test_equals_oracle_uniform(gn, oracle, n, d, nq, k):
    rng = np.random.default_rng(n + d)
    _check(gn, oracle, rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32), k, sub=300)


@pytest.mark.parametrize("shuffle", [True, False])
def test_clusters(gn, oracle, shuffle):
    """Cluster after cluster in the database, or mixed."""
    rng = np.random.default_rng(7)
    c = rng.standard_normal((200, 64)).astype(np.float32)
    comp = np.repeat(np.arange(200), 400)
    if shuffle:
        rng.shuffle(comp)
    db = (c[comp] + 0.2 * rng.standard_normal((len(comp), 64))).astype(np.float32)
    q = (c[rng.integers(0, 200, 600)] + 0.2 * rng.standard_normal((600, 64))).astype(np.float32)
    _check(gn, oracle, db, q, 10)


@pytest.mark.parametrize("case", ["offset", "large offset", "tiny", "duplicates", "few values", "scales"])
def test_data_that_the_bound_cannot_separate(gn, oracle, case):
    rng = np.random.default_rng(11)
    n, d, nq = 50_000, 48, 700
    db, q = rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32)
    if case == "offset":
        db, q = db + np.float32(100), q + np.float32(100)
    elif case == "large offset":
        db, q = db + np.float32(1e4), q + np.float32(1e4)
    elif case == "tiny":
        db, q = db * np.float32(1e-20), q * np.float32(1e-20)
    elif case == "duplicates":
        db = db[rng.integers(0, 60, n)]
    elif case == "few values":
        db, q = np.round(db[:, :] * 1), np.round(q * 1)
    else:
        db *= np.float32(10) ** rng.integers(-6, 7, (n, 1)).astype(np.float32)
    _check(gn, oracle, db.astype(np.float32), q.astype(np.float32), 10, sub=250)


@pytest.mark.parametrize("where", ["rows", "queries", "both"])
def test_values_that_are_not_finite(gn, where):
    """Against the same search in parts too small for this path."""
    rng = np.random.default_rng(13)
    db, q = rng.random((40_000, 40), dtype=np.float32), rng.random((1024, 40), dtype=np.float32)
    if where != "queries":
        db[5::97, 3] = np.inf
        db[6::89, 7] = np.nan
        db[100, 5] = 1e30
    if where != "rows":
        q[3, 2] = np.inf
        q[700, 0] = np.nan
        q[9, 1] = 1e30
    ix = gn.FlatL2Index()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, 10)
    parts = [ix.search_knn_arrays(q[i:i + 32], 10) for i in range(0, 1024, 32)]
    assert np.array_equal(idx, np.concatenate([p[0] for p in parts]))
    assert np.array_equal(dist.view(np.uint32), np.concatenate([p[1] for p in parts]).view(np.uint32))


def test_new_rows_replace_the_old_ones(gn, oracle):
    rng = np.random.default_rng(17)
    ix = gn.FlatL2Index()
    for n, d in ((40_000, 64), (60_000, 64), (40_000, 30)):
        db, q = rng.random((n, d), dtype=np.float32), rng.random((1400, d), dtype=np.float32)
        ix.set(db)
        idx, dist = ix.search_knn_arrays(q, 6)
        oi, od = oracle.knn_float("l2", db, q[:200], 6)
        assert np.array_equal(idx[:200], oi) and np.array_equal(dist[:200].view(np.uint32), od.view(np.uint32))
