"""Device-pointer calls under stream capture (needs a B200): the exact scan's
workspace becomes an allocation of the graph, the beam takes nothing.  A graph
replayed on new queries gives what a direct call gives, bit for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import _capi, pickling

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 40])
def test_exact_scan_replays(tmp_path, nq):
    n, dim, k = 5000, 40, 10
    rng = np.random.default_rng(nq)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    (tmp_path / "bf.bin").write_bytes(pickling.bf_rows_to_file(x, np.arange(n, dtype=np.uint64), n, dim))
    g = H.BFIndex("l2", dim)
    g.load_index(str(tmp_path / "bf.bin"))
    q = [torch.from_numpy(rng.standard_normal((nq, dim)).astype(np.float32)).cuda() for _ in range(3)]
    dq = q[0].clone()
    lab = torch.zeros(nq, k, dtype=torch.int64, device="cuda")
    dist = torch.zeros(nq, k, device="cuda")
    cnt = torch.zeros(nq, dtype=torch.int32, device="cuda")
    opts = _capi.SearchOpts()
    opts.flags = _capi.DEVICE_PTRS

    def call(stream):
        opts.stream = stream.cuda_stream
        _capi.check(_capi.lib().hnswgpu_search(g._h, C.c_void_p(dq.data_ptr()), nq, k, C.byref(opts),
                                               C.c_void_p(lab.data_ptr()), C.c_void_p(dist.data_ptr()),
                                               C.c_void_p(cnt.data_ptr())))

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    call(s)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(s)
    for j in (1, 2, 1):
        want = g.knn_query(q[j].cpu().numpy(), k)
        dq.copy_(q[j])
        lab.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(lab.cpu().numpy().astype(np.uint64), want[0].astype(np.uint64))
        assert np.array_equal(dist.cpu().numpy().view(np.uint32), want[1].view(np.uint32))
        assert bool((cnt == k).all())
