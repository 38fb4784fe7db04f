"""The bound that a tensor-core scan takes from its pilot launch, over and over on the
same data: the row norms that the pilot reads sit in a ring of slots that bulk copies
refill, and a slot refilled too early gives queries a bound that is too low.  Shapes
with several units of few tiles per block, where the next unit's norms follow closely."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq", [(10_000, 128, 8192), (10_000, 100, 20_000), (24_000, 128, 16_384)])
def test_shortlist_is_the_same_every_time(gn, n, d, nq):
    """k equal to the shortlist: a bound below the k-th score loses results."""
    rng = np.random.default_rng(n + d)
    ix = gn.FlatL2TCIndex(shortlist=32)
    ix.set(rng.random((n, d), dtype=np.float32))
    q = rng.random((nq, d), dtype=np.float32)
    idx, dist = ix.search_knn_arrays(q, 32)
    assert (idx >= 0).all()
    for _ in range(30):
        again = ix.search_knn_arrays(q, 32)
        assert np.array_equal(idx, again[0]) and np.array_equal(dist, again[1])


def test_exact_l2_keeps_to_the_tensor_cores(gn):
    """Well separated rows: no batch needs the FP32 scan (a bound that is too low
    leaves fewer candidates than results, which hands the batch over to it)."""
    from pynear_gb300 import _lib
    rng = np.random.default_rng(5)
    ix = gn.FlatL2Index()
    ix.set(rng.random((10_000, 32), dtype=np.float32))
    q = rng.random((20_000, 32), dtype=np.float32)
    lib, name = _lib.load(), ctypes.create_string_buffer(64)
    lib.gn_timing_enable(1)
    try:
        for _ in range(40):
            ix.search_knn_arrays(q, 10)
        _lib.check(lib.gn_timing_last(None, name, 64))
    finally:
        lib.gn_timing_enable(0)
    assert name.value == b"tc_topk_kernel"
