"""Tensor-core shortlist over small databases, on both sides of the pilot's least rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 300, 700, 1024, 4096, 16_384, 20_011, 32_767, 32_768])
@pytest.mark.parametrize("precision", ["bf16", "fp8"])
def test_small_databases_equal_the_exact_scan(gn, n, precision):
    rng = np.random.default_rng(n)
    db = rng.standard_normal((n, 70), dtype=np.float32)
    ix = gn.FlatL2TCIndex(shortlist=56 if precision == "fp8" else 40, precision=precision)
    ix.set(db)
    ex = gn.FlatL2Index()
    ex.set(db)
    for nq in (1, 130, 1500):
        q = rng.standard_normal((nq, 70), dtype=np.float32)
        idx, dist = ix.search_knn_arrays(q, 1)
        ei, ed = ex.search_knn_arrays(q, 1)
        same = (idx == ei).mean()
        assert same >= (0.99 if precision == "fp8" else 1.0)
        assert np.array_equal(dist[idx == ei], ed[idx == ei])


@pytest.mark.parametrize("n,nbytes,nq,k", [(4095, 512, 4000, 5), (4096, 512, 4000, 1), (4200, 511, 4000, 64),
                                           (20_011, 64, 6300, 10)])
def test_hamming_over_small_databases(gn, oracle, n, nbytes, nq, k):
    rng = np.random.default_rng(n + k)
    db = rng.integers(0, 256, (n, nbytes), dtype=np.uint8)
    db[n // 2 :] = db[: n - n // 2]
    q = rng.integers(0, 256, (nq, nbytes), dtype=np.uint8)
    ix = gn.FlatHammingIndex()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    oi, od = oracle.knn_hamming(db, q[:200], k)
    assert np.array_equal(idx[:200], oi) and np.array_equal(dist[:200], od)
    oi, od = oracle.knn_hamming(db, q[-100:], k)
    assert np.array_equal(idx[-100:], oi) and np.array_equal(dist[-100:], od)


@pytest.mark.parametrize("n,d,nq,k", [(4095, 1024, 500, 5), (4096, 1024, 500, 1), (4300, 2000, 300, 32),
                                      (20_011, 70, 1500, 10)])
def test_exact_l2_over_small_databases(gn, oracle, n, d, nq, k):
    rng = np.random.default_rng(n + d)
    db = rng.standard_normal((n, d), dtype=np.float32)
    db[n // 2 :] = db[: n - n // 2]
    q = rng.standard_normal((nq, d), dtype=np.float32)
    ix = gn.FlatL2Index()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    oi, od = oracle.knn_float("l2", db, q[:64], k)
    assert np.array_equal(idx[:64], oi) and np.array_equal(dist[:64].view(np.uint32), od.view(np.uint32))


def test_hamming_of_few_words(gn, oracle):
    rng = np.random.default_rng(4)
    db = rng.integers(0, 256, (31_361, 20), dtype=np.uint8)
    q = rng.integers(0, 256, (3585, 20), dtype=np.uint8)
    ix = gn.FlatHammingIndex()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, 3)
    oi, od = oracle.knn_hamming(db, q, 3)
    assert np.array_equal(idx, oi) and np.array_equal(dist, od)
