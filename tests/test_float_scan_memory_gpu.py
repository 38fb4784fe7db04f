"""Device memory of a large float batch with many results: about that of its results,
whatever the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["FlatL1Index", "FlatL2Index"])
def test_scratch_of_a_large_batch_is_bounded(gn, oracle, kind):
    import torch
    torch.zeros(1, device="cuda")
    rng = np.random.default_rng(1)
    db, q, k = rng.random((4096, 5), dtype=np.float32), rng.random((150_000, 5), dtype=np.float32), 100
    ix = getattr(gn, kind)()
    ix.set(db)
    ix.search_knn_arrays(q[:100], k)  # kernels loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    idx, dist = ix.search_knn_arrays(q, k)
    used = free - torch.cuda.mem_get_info()[0]
    results = len(q) * k * 12
    # a list of k keys per query was the scan's scratch before it had buffers; 128 MB: one block of queries
    assert used <= results + len(q) * k * 8 + (128 << 20)
    for s in (slice(0, 60), slice(74_990, 75_050), slice(len(q) - 60, None)):
        oi, od = oracle.knn_float("l1" if kind == "FlatL1Index" else "l2", db, q[s], k)
        assert np.array_equal(idx[s], oi) and np.array_equal(dist[s].view(np.uint32), od.view(np.uint32))
