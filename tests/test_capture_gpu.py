"""Other threads while a thread captures a CUDA graph in the default ("global")
mode, in which a memory call of any thread ends the capture unless that thread
asks otherwise: the end of a thread that called a solver, which frees its
pinned words, must leave the capture alone."""
import threading

import numpy as np
import pytest

from flashx_b200 import sparse_matrix
from flashx_b200.algs import PageRank

pytestmark = pytest.mark.gpu


def test_capture_beside_an_ending_thread(torch_cuda):
    torch = torch_cuda
    n = 30000
    rng = np.random.default_rng(1)
    s, d = (torch.from_numpy(rng.integers(0, n, 200000).astype(np.int32)).cuda() for _ in range(2))
    m = sparse_matrix.from_device_edges(s, d, None, nrows=n, ncols=n, dedup=True, transpose=True)
    x = torch.randn((n, 16), device="cuda")
    y = torch.empty_like(x)
    assert m.multiply(x, y)
    want = y.clone()
    ready, go = threading.Event(), threading.Event()

    def work():
        PageRank(m, 5, 0.85)
        torch.cuda.synchronize()
        ready.set()
        go.wait()

    t = threading.Thread(target=work)
    t.start()
    ready.wait()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert m.multiply(x, y)
        go.set()
        t.join()
        assert m.multiply(x, y)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
