"""Edges of the k-means kernels against the oracle: rows around a block's
step and chunk, tails of eight coordinates, cluster slabs, duplicated rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(3, 1, 3), (127, 2, 5), (128, 3, 9), (129, 4, 17), (257, 5, 8), (1000, 6, 11),
                                   (1025, 7, 40), (4097, 8, 33), (131_073, 13, 12), (262_145, 20, 6), (999, 515, 7)])
def test_float_seeds_equal_the_serial_rule(gn, oracle, n, d, k):
    """max_iter 0 returns the seeds, bit for bit the oracle's serial loop."""
    data = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    _, cent = gn.kmeans_l2(data, k, 0, 42)
    _, ocent, _ = oracle.kmeans_l2(data, k, 0, 42)
    assert np.array_equal(cent.view(np.uint32), ocent.view(np.uint32))


@pytest.mark.parametrize("n,nbytes,nlist,iters,distinct", [
    (2, 1, 2, 20, None), (255, 5, 2, 20, None), (257, 16, 31, 20, None), (4099, 33, 61, 20, None),
    (20_001, 8, 1025, 3, None),       # a second slab of clusters in the bit counts
    (525_313, 4, 9, 2, None),         # chunks longer than one step of rows
    (2000, 12, 60, 20, 40),           # more lists than distinct rows: the draws' total reaches zero
    (70_000, 7700, 6, 1, None),       # totals past 32 bits: the host draws
])
def test_binary_build_equals_the_oracle(gn, oracle, n, nbytes, nlist, iters, distinct):
    rng = np.random.default_rng(n + nbytes)
    db = rng.integers(0, 256, (distinct or n, nbytes), dtype=np.uint8)
    if distinct:
        db = np.repeat(db, n // distinct, axis=0)
    ix = gn.IVFFlatBinaryIndex(nlist=nlist, nprobe=1, max_iter=iters)
    ix.set(db)
    cent, labels = ix.export()
    oc, ol = oracle.ivfbin_build(db, nlist, iters)
    assert np.array_equal(cent, oc) and np.array_equal(labels, ol)


@pytest.mark.parametrize("n,d,k,distinct", [(300, 3, 9, 5), (2000, 16, 40, 7), (152 * 33 + 1, 8, 12, 3), (5000, 64, 300, None)])
def test_float_seeds_where_the_serial_sum_decides(gn, oracle, n, d, k, distinct):
    """Fewer distinct rows than centroids: the later draws' distances are all zero,
    and a draw of the first ones may fall on a boundary between equal rows."""
    rng = np.random.default_rng(n + k)
    data = rng.standard_normal((distinct or n, d)).astype(np.float32)
    if distinct:
        data = data[rng.integers(0, distinct, n)]
    _, cent = gn.kmeans_l2(data, k, 0, 42)
    _, ocent, _ = oracle.kmeans_l2(data, k, 0, 42)
    assert np.array_equal(cent.view(np.uint32), ocent.view(np.uint32))
