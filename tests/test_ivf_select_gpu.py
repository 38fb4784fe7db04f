"""Selection stage of the tensor-core IVF engine: the launch shapes that the
batch size picks, and its exact distances against float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gn():
    import pynear_gb300

    return pynear_gb300


def _exact(q, x):
    """The sum of the squared FP32 differences (each rounded, as the kernel's), in float64."""
    return ((q - x).astype(np.float64) ** 2).sum(-1)


def _index(gn, rows, d, n_probe, shortlist=40, seed=0):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((150, d), dtype=np.float32)
    db = c[rng.integers(0, 150, rows)] + np.float32(0.4) * rng.standard_normal((rows, d), dtype=np.float32)
    q = c[rng.integers(0, 150, 4300)] + np.float32(0.4) * rng.standard_normal((4300, d), dtype=np.float32)
    ix = gn.IVFFlatL2Index(n_clusters=96, n_probe=n_probe, engine="tc", shortlist=shortlist)
    ix.set(db)
    return ix, db, q


# one, two, four and eight warps per query: 28 warps fit each of 152 SMs; more than 64
# probes are laid out in turns, and 20,000 rows in 96 lists give more than 128 slots
@pytest.mark.parametrize("n_probe", [5, 90])
def test_batch_sizes_agree(gn, n_probe):
    ix, db, q = _index(gn, 20_000, 24, n_probe)
    t = np.zeros((7, 4), np.int32)
    t[:, 2] = 32
    ix.tuning = t
    ref = ix.search_knn_arrays(q, 10)
    ix.tuning = np.zeros((7, 4), np.int32)
    for nq in (1, 532, 533, 1064, 1065, 2128, 2129, 4256, 4257):
        for a, b in zip(ix.search_knn_arrays(q[:nq], 10), ref):
            np.testing.assert_array_equal(a, b[:nq])


# the sum's own error is far below the last rounding: half an ulp and a little, so one
# ulp (2^-23 at most) is allowed; dimensions across the 4, 128 and 512 column blocks
@pytest.mark.parametrize("d", [1, 3, 37, 128, 130, 512, 515, 1030])
@pytest.mark.parametrize("shortlist", [16, 64])
def test_distances_are_correctly_rounded_sums(gn, d, shortlist):
    ix, db, q = _index(gn, 3000, d, 8, shortlist, seed=d)
    for nq in (3, 3000):
        idx, dist, cnt = ix.search_knn_arrays(q[:nq], 10)[:3]
        assert (idx >= 0).all()
        want = _exact(q[:nq, None, :], db[idx])
        assert (np.abs(dist - want) <= want * 2.0**-23).all()


def test_distances_near_the_largest_float(gn):
    """Squares whose sum fits a float but not twice over."""
    n = 400
    db = np.zeros((n, 8), np.float32)
    db[:, 0] = np.linspace(1.30e19, 1.32e19, n, dtype=np.float32)
    db[:, 1] = np.linspace(1e18, 2e18, n, dtype=np.float32)
    ix = gn.IVFFlatL2Index(n_clusters=4, n_probe=4, engine="tc")
    ix.set(db)
    q = np.zeros((2, 8), np.float32)
    idx, dist, cnt = ix.search_knn_arrays(q, 10)[:3]
    want = _exact(q[:, None, :], db[idx])
    assert np.isfinite(dist).all()
    assert (np.abs(dist - want) <= want * 2.0**-23).all()
