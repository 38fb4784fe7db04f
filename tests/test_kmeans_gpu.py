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


@pytest.mark.parametrize("n,d,k", [(70, 3, 1), (513, 16, 127), (20_000, 20, 128), (19_457, 33, 129), (4100, 64, 255),
                                   (40_001, 80, 256), (3000, 100, 256), (3000, 7, 300)])
def test_labels_are_nearest_centroids(gn, n, d, k):
    """One assignment, around 128 and 256 centroids and blocks of rows that end inside a
    tile.  A score's error is at most (d + 3) 2^-24 (2 |x| |c| + |c|^2)."""
    data = np.random.default_rng(n + k).standard_normal((n, d)).astype(np.float32)
    _, seeds = gn.kmeans_l2(data, k, 0, 42)
    labels, _ = gn.kmeans_l2(data, k, 1, 42)
    x, c = data.astype(np.float64), np.asarray(seeds, np.float64)
    cn = (c**2).sum(1)
    score = cn - 2 * x @ c.T
    err = (d + 3) * 2.0**-24 * (2 * np.sqrt((x**2).sum(1).max() * cn.max()) + cn.max())
    assert (score[np.arange(n), labels] <= score.min(1) + 2 * err).all()


@pytest.mark.parametrize("k", [5, 128, 256])
def test_labels_where_scores_overflow(gn, k):
    """Products that overflow (scores of +-inf and NaN): 240 zero columns more take the
    labels to the other assignment kernel and change no sum."""
    rng = np.random.default_rng(k)
    data = (rng.integers(0, 2, (900, 16)) * 2 - 1).astype(np.float32) * np.float32(1e30)
    data[::3] = rng.standard_normal((300, 16)).astype(np.float32)
    labels = gn.kmeans_l2(data, k, 1, 42)[0]
    wide = gn.kmeans_l2(np.pad(data, ((0, 0), (0, 240))), k, 1, 42)[0]
    assert np.array_equal(labels, wide)
