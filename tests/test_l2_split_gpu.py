"""Exact L2 on the tensor cores for values that lose most when they are split into two
BF16 parts: every coordinate half a BF16 step above a BF16 value and of one sign, so
that what is left out adds up, with rows a few FP32 steps apart around every place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq,k", [(20_000, 64, 1300, 10), (40_000, 48, 900, 32), (9_000, 170, 1100, 5)])
def test_values_that_round_worst(gn, oracle, n, d, nq, k):
    rng = np.random.default_rng(n + d)

    def worst(m):
        v = 1 + (2 * rng.integers(0, 128, (m, d)) + 1) * 2.0**-8  # ties between two BF16 values
        return (v * (1 + rng.integers(-8, 9, (m, d)) * 2.0**-16)).astype(np.float32)

    db = worst(n // 4)
    near = np.concatenate([db] + [db.copy() for _ in range(3)])
    cols = rng.integers(0, d, len(near))
    near[np.arange(len(near)), cols] = np.nextafter(near[np.arange(len(near)), cols], np.float32(4))
    db = near[rng.permutation(len(near))]
    q = worst(nq)
    ix = gn.FlatL2Index()
    ix.set(db)
    for _ in range(2):
        idx, dist = ix.search_knn_arrays(q, k)
        oi, od = oracle.knn_float("l2", db, q[:200], k)
        assert np.array_equal(idx[:200], oi) and np.array_equal(dist[:200].view(np.uint32), od.view(np.uint32))
