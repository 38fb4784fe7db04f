"""Which scan answers exact L2 batches: one odd batch does not keep an index off the
tensor cores, rows that they cannot separate do."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Route:
    """The kernel that the last search ran."""

    def __init__(self):
        from pynear_gb300 import _lib
        self.lib = _lib.load()

    def __enter__(self):
        self.lib.gn_timing_enable(1)
        return self

    def __exit__(self, *exc):
        self.lib.gn_timing_enable(0)

    def __call__(self, ix, q, k=10):
        from pynear_gb300 import _lib
        ix.search_knn_arrays(q, k)
        name = ctypes.create_string_buffer(64)
        _lib.check(self.lib.gn_timing_last(None, name, 64))
        return name.value.decode()


@pytest.fixture
def rows():
    rng = np.random.default_rng(3)
    return rng.random((60_000, 40), dtype=np.float32), rng.random((2048, 40), dtype=np.float32)


def test_an_odd_batch_costs_that_batch(gn, rows):
    db, q = rows
    ix = gn.FlatL2Index()
    ix.set(db)
    odd = q.copy()
    odd[7, 3] = np.nan
    with _Route() as route:
        for _ in range(4):
            route(ix, q)
        assert route(ix, q) == "tc_topk_kernel"
        for batch in (odd, q, odd, odd, q):
            assert route(ix, batch) == "tc_topk_kernel"
        for _ in range(8):
            route(ix, odd)
        assert route(ix, q) == "float_scan_kernel"
        assert any(route(ix, q) == "tc_topk_kernel" for _ in range(40))
        assert route(ix, q) == "tc_topk_kernel"


def test_rows_that_never_fit_are_left_to_the_float_scan(gn, rows):
    db, q = rows
    ix = gn.FlatL2Index()
    ix.set(np.repeat(db[:1], len(db), axis=0))  # more rows at one distance than the buffers hold
    with _Route() as route:
        for _ in range(12):
            route(ix, q)
        names = [route(ix, q) for _ in range(64)]
        assert names.count("tc_topk_kernel") <= 2
        ix.set(db)
        for _ in range(4):
            route(ix, q)
        assert route(ix, q) == "tc_topk_kernel"
