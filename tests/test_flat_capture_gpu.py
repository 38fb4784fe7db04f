"""Flat searches captured into a CUDA graph: large batches, whose usual route keeps a
copy of the rows, answer from the rows that are there when the graph is replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,d,nq,k", [("l2", 60_000, 64, 2000, 10), ("l2", 50_000, 30, 1500, 100),
                                           ("hamming", 40_000, 64, 4096, 10), ("hamming", 40_000, 20, 4096, 33)])
def test_a_captured_search_sees_new_rows(gn, kind, n, d, nq, k):
    import torch
    from pynear_gb300 import _lib
    rng = np.random.default_rng(n + k)
    ham = kind == "hamming"
    cls = gn.FlatHammingIndex if ham else gn.FlatL2Index

    def data(m):
        return rng.integers(0, 256, (m, d), dtype=np.uint8) if ham else rng.random((m, d), dtype=np.float32)

    ix, rows, q = cls(), [data(n) for _ in range(3)], data(nq)
    pitch = (d + 15) // 16 * 16 if ham else (d + 3) // 4 * 4
    dq = torch.zeros((nq, pitch), dtype=torch.uint8 if ham else torch.float32, device="cuda")
    dq[:, :d] = torch.from_numpy(q)
    idx = torch.empty((nq, k), dtype=torch.int64, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.int64 if ham else torch.float32, device="cuda")
    stream = torch.cuda.Stream()

    def search():
        _lib.call("gn_flat_search_knn_device", ix._h.h, dq.data_ptr(), nq, k, idx.data_ptr(), dist.data_ptr(),
                  stream.cuda_stream)

    def check(r):
        other = cls()
        other.set(r)
        oi, od = other.search_knn_arrays(q, k)
        assert np.array_equal(idx.cpu().numpy(), oi) and np.array_equal(dist.cpu().numpy(), od)

    ix.set(rows[0])
    for _ in range(4):
        search()
    stream.synchronize()
    check(rows[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        search()
    for r in rows:
        ix.set(r)
        idx.zero_()
        graph.replay()
        torch.cuda.synchronize()
        check(r)
    search()  # and uncaptured again
    stream.synchronize()
    check(rows[-1])
