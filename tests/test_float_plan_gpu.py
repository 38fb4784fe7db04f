"""Shapes at the edges of the float scan's plan: fewer rows than a stage or a warp takes,
in narrow and wide rows, and batches of a little more than the GPU takes at once (the
whole wave first, then the rest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = {"l2": "FlatL2Index", "l1": "FlatL1Index", "linf": "FlatChebyshevIndex"}


def _check(gn, oracle, metric, n, d, nq, k, subs):
    rng = np.random.default_rng(n * 7 + d)
    db, q = rng.standard_normal((n, d), dtype=np.float32), rng.standard_normal((nq, d), dtype=np.float32)
    if n > 3:
        db[n // 2] = db[0]
    ix = getattr(gn, KINDS[metric])()
    ix.set(db)
    idx, dist = ix.search_knn_arrays(q, k)
    for s in subs:
        oi, od = oracle.knn_float(metric, db, q[s], k)
        assert np.array_equal(idx[s], oi) and np.array_equal(dist[s].view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 95, 97, 127, 129, 160, 255, 257])
@pytest.mark.parametrize("d", [1, 3, 31, 32, 33, 130, 700])
def test_few_rows(gn, oracle, metric, n, d):
    for nq in (1, 3, 7, 40):
        _check(gn, oracle, metric, n, d, nq, min(n, 9), [slice(0, 40)])


@pytest.mark.parametrize("metric", ["l2", "l1"])
@pytest.mark.parametrize("n,d,nq,k", [(3000, 32, 9000, 10), (3500, 40, 7297, 5), (3500, 40, 7296, 5), (5000, 32, 14_591, 1),
                                      (2500, 65, 8000, 64), (20_000, 8, 7500, 33), (3001, 33, 7312, 65)])
def test_a_little_more_than_a_wave(gn, oracle, metric, n, d, nq, k):
    _check(gn, oracle, metric, n, d, nq, k, [slice(0, 30), slice(7280, 7320), slice(nq - 30, nq)])
