"""The largest ef a search takes (needs a B200): a fixed function of the
dimension, the tie order, the filter and the precision, and searches at it work."""
import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import _capi
from oracle import oracle as O
from test_gpu_graph_forms import write_graph

pytestmark = pytest.mark.gpu

# dim, order, precision, filtered: largest ef
LIMITS = [
    (285, "id", "fp32", False, 27598), (285, "id", "fp32", True, 5519), (400, "id", "fp32", False, 27670),
    (400, "reference", "fp32", False, 4595), (400, "reference", "fp32", True, 2757), (500, "id", "fp32", True, 5530),
    (7, "id", "fp32", False, 28714), (16, "reference", "fp32", False, 4758), (128, "id", "bf16", False, 28206),
    (3000, "id", "fp32", False, 25908), (20000, "reference", "fp32", False, 1467),
]


@pytest.mark.parametrize("dim,order,prec,filtered,limit", LIMITS)
def test_limit(tmp_path, dim, order, prec, filtered, limit):
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((60, dim)).astype(np.float32)
    labels = write_graph(tmp_path / "g.bin", x, "l2", 8)
    g = H.Index("l2", dim)
    g.load_index(str(tmp_path / "g.bin"))
    g.precision = prec
    q = rng.standard_normal((5, dim)).astype(np.float32)
    filt = (lambda v: v % 2 == 0) if filtered else None
    got = g.knn_query_traced(q, 10, ef=limit, tie_order=order, filter=filt)
    allow = np.array([v % 2 == 0 for v in labels], np.uint8) if filtered else None
    want = O.Hnsw(str(tmp_path / "g.bin"), "l2", dim).search(
        q, 10, limit, mode=O.REFERENCE if order == "reference" else O.CANONICAL, allow=allow)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    with pytest.raises(_capi.HnswGpuError, match="ef too large"):
        g.knn_query_traced(q, 10, ef=limit + 1, tie_order=order, filter=filt)
