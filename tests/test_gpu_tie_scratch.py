"""Tie-exact searches share an index's candidate-heap tails (needs a B200):
calls on several streams, and captured calls replayed after larger batches and
larger ef, return what the same calls return alone, bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import _capi
from test_gpu_graph_forms import write_graph

pytestmark = pytest.mark.gpu

DIM = 16


@pytest.fixture(scope="module")
def ties(tmp_path_factory):
    """Rows that tie so often that most queries repeat with the heaps."""
    path = tmp_path_factory.mktemp("ties") / "g.bin"
    rng = np.random.default_rng(3)
    write_graph(path, rng.integers(0, 4, (3000, DIM)).astype(np.float32), "l2", 16)
    return path, rng.integers(0, 4, (4000, DIM)).astype(np.float32)


class Call:
    """One asynchronous search with its own device buffers."""

    def __init__(self, g, q, k, ef, flags=0):
        self.g, self.k, self.q = g, k, torch.from_numpy(q).cuda()
        self.lab = torch.zeros(len(q), k, dtype=torch.int64, device="cuda")
        self.dist = torch.zeros(len(q), k, device="cuda")
        self.cnt = torch.zeros(len(q), dtype=torch.int32, device="cuda")
        self.o = _capi.SearchOpts()
        self.o.flags = _capi.DEVICE_PTRS | _capi.EXACT_TIES | flags
        self.o.ef = ef

    def __call__(self, stream):
        self.o.stream = stream.cuda_stream
        _capi.check(_capi.lib().hnswgpu_search(self.g._h, C.c_void_p(self.q.data_ptr()), len(self.q), self.k,
                                               C.byref(self.o), C.c_void_p(self.lab.data_ptr()),
                                               C.c_void_p(self.dist.data_ptr()), C.c_void_p(self.cnt.data_ptr())))

    def same(self, want):
        return np.array_equal(self.lab.cpu().numpy().astype(np.uint64), want[0]) and \
            np.array_equal(self.dist.cpu().numpy(), want[1])


def load(path):
    g = H.Index("l2", DIM)
    g.load_index(str(path))
    return g


def test_streams(ties):
    path, q = ties
    g = load(path)
    shapes = [(10, 64), (10, 16), (30, 100)]
    want = {s: [a.copy() for a in g.knn_query_traced(q, s[0], ef=s[1], tie_order="replay")[:2]] for s in shapes}
    streams = [torch.cuda.Stream() for _ in range(3)]
    calls = []
    torch.cuda.synchronize()
    for i in range(12):
        s = shapes[i % 3]
        lo = 1000 * (i % 2)
        c = Call(g, q[lo:lo + 2500], *s, flags=_capi.REPLAY_ALL if i % 4 == 3 else 0)
        torch.cuda.synchronize()
        calls.append((c, s, lo))
    for i, (c, s, lo) in enumerate(calls):
        c(streams[i % 3])
        if i % 5 == 4:  # a host call between them
            got = g.knn_query_traced(q[:1500], 10, ef=64, tie_order="reference")
            assert np.array_equal(got[0], want[shapes[0]][0][:1500])
    torch.cuda.synchronize()
    for c, s, lo in calls:
        assert c.same((want[s][0][lo:lo + 2500], want[s][1][lo:lo + 2500]))
    assert g.get_status() == 0


@pytest.mark.parametrize("nq", [50, 2500])
def test_captured_call_outlives_larger_ones(ties, nq):
    path, q = ties
    g = load(path)
    ef, k = 48, 10
    want = [a[:nq] for a in load(path).knn_query_traced(q, k, ef=ef, tie_order="replay")[:2]]
    s = torch.cuda.Stream()
    c = Call(g, q[:nq], k, ef)
    torch.cuda.synchronize()
    Call(g, q[:50], k, ef)(s)  # a small batch provides the scratch of any
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        c(s)
    for shape in ((4000, ef), (60, 200), (4000, 300)):
        g.knn_query_traced(q[:shape[0]], k, ef=shape[1], tie_order="reference")
        c.lab.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert c.same(want)


def test_capture_without_scratch_is_refused(ties):
    path, q = ties
    g = load(path)
    c = Call(g, q[:50], 10, 48)
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with pytest.raises(_capi.HnswGpuError, match="before capturing"):
        with torch.cuda.graph(graph, stream=s):
            c(s)
    c(s)
    s.synchronize()
    assert c.same([a[:50] for a in g.knn_query_traced(q, 10, ef=48, tie_order="replay")[:2]])
