"""Which scan answers the first exact L2 searches of new rows: the split rows that the
tensor cores want are made once enough searches of the same rows can use them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nq,at_once", [(40_000, 64, 700, False), (300_000, 128, 64, False),
                                            (60_000, 64, 4096, True)])
def test_new_rows_are_split_when_it_pays(gn, oracle, n, d, nq, at_once):
    from pynear_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(n)
    ix = gn.FlatL2Index()
    lib.gn_timing_enable(1)
    try:
        for _ in range(2):  # a second set() starts anew
            db, q = rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32)
            ix.set(db)
            names = []
            for i in range(40):
                idx, dist = ix.search_knn_arrays(q, 10)
                name = ctypes.create_string_buffer(64)
                _lib.check(lib.gn_timing_last(None, name, 64))
                names.append(name.value.decode())
                if i == 0:
                    first = idx, dist
            assert np.array_equal(first[0], idx) and np.array_equal(first[1], dist)
            oi, od = oracle.knn_float("l2", db, q[:50], 10)
            assert np.array_equal(idx[:50], oi) and np.array_equal(dist[:50].view(np.uint32), od.view(np.uint32))
            assert names[0] == ("tc_topk_kernel" if at_once else "float_scan_kernel")
            assert names[-1] == "tc_topk_kernel"
    finally:
        lib.gn_timing_enable(0)
