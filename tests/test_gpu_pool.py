"""What an index keeps of its calls' workspaces (needs a B200): a bounded
amount, whatever the largest call took."""
import ctypes as C

import numpy as np
import pytest
import torch

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import _capi, pickling

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_large_call_gives_its_memory_back(tmp_path):
    n, dim, k, nq = 200, 128, 4, 1 << 20
    rng = np.random.default_rng(0)
    x = pickling.normalize_rows(rng.standard_normal((n, dim)).astype(np.float32))
    (tmp_path / "bf.bin").write_bytes(pickling.bf_rows_to_file(x, np.arange(n, dtype=np.uint64), n, dim))
    g = H.BFIndex("cosine", dim)
    g.load_index(str(tmp_path / "bf.bin"))
    q = torch.randn(nq, dim, device="cuda")
    lab = torch.zeros(nq, k, dtype=torch.int64, device="cuda")
    dist = torch.zeros(nq, k, device="cuda")
    cnt = torch.zeros(nq, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    o = _capi.SearchOpts()
    o.flags = _capi.DEVICE_PTRS
    o.stream = s.cuda_stream

    def call(m):
        _capi.check(_capi.lib().hnswgpu_search(g._h, C.c_void_p(q.data_ptr()), m, k, C.byref(o),
                                               C.c_void_p(lab.data_ptr()), C.c_void_p(dist.data_ptr()),
                                               C.c_void_p(cnt.data_ptr())))
        s.synchronize()

    torch.cuda.synchronize()
    g.knn_query(x[:4], k)  # the kernels are loaded, the pool exists
    free0 = torch.cuda.mem_get_info()[0]
    call(nq)  # 512 MB of normalised queries and 64 MB of keys
    call(8)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 288 * MB  # 256 MB and a block's rounding
    assert np.array_equal(lab[:8].cpu().numpy().astype(np.uint64), g.knn_query(q[:8].cpu().numpy(), k)[0])
