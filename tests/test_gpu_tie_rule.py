"""Reference order on graphs where a neighbour is rejected at a lowerBound that
an earlier neighbour of its own list has lowered while two candidates tie (needs
a B200): the smallest such graph, and many queries over small-integer rows
against the replay of the heaps for every query."""
import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import pickling
from oracle import oracle as O
from test_gpu_graph_forms import write_graph

pytestmark = pytest.mark.gpu

LINKS = [[5, 1, 7, 6, 4], [4, 6, 5, 7, 0], [6, 3, 4, 0, 5], [4, 7, 6, 2, 0],
         [0, 2, 3, 6, 7], [4, 7, 1, 6, 0], [3, 4, 1, 2, 0], [6, 4, 5, 1, 0]]
DIST = [1, 2, 1, 1, 0, 2, 0, 2]  # squared, to the zero query; entry 0


def write_small(path, dim, M):
    n, M0 = len(LINKS), 2 * M
    x = np.zeros((n, dim), np.float32)
    for i, d in enumerate(DIST):
        x[i, :d] = 1
    size = 4 + 4 * M0 + 4 * dim + 8
    rec = np.zeros((n, size), np.uint8)
    for i, l in enumerate(LINKS):
        head = np.zeros(1 + M0, np.uint32)
        head[0] = len(l)
        head[1:1 + len(l)] = l
        rec[i, :4 + 4 * M0] = head.view(np.uint8)
    rec[:, 4 + 4 * M0:-8] = x.view(np.uint8).reshape(n, -1)
    rec[:, -8:] = np.arange(n, dtype=np.uint64).view(np.uint8).reshape(n, 8)
    state = dict(offset_level0=0, max_elements=n, cur_element_count=n, size_data_per_element=size,
                 label_offset=size - 8, offset_data=4 + 4 * M0, max_level=0, enterpoint_node=0, max_M=M, max_M0=M0,
                 M=M, mult=1 / np.log(M), ef_construction=100, size_links_per_element=4 + 4 * M,
                 element_levels=np.zeros(n, np.int32), data_level0=rec.reshape(-1), link_lists=np.zeros(0, np.uint8))
    path.write_bytes(pickling.state_to_file_bytes(state))


@pytest.mark.parametrize("dim,M", [(4, 4), (7, 4), (16, 8), (33, 16), (48, 32)])
def test_smallest_graph(tmp_path, dim, M):
    write_small(tmp_path / "g.bin", dim, M)
    o = O.Hnsw(str(tmp_path / "g.bin"), "l2", dim)
    g = H.Index("l2", dim)
    g.load_index(str(tmp_path / "g.bin"))
    q = np.zeros((1, dim), np.float32)
    assert set(o.search(q, 4, 4, mode=O.REFERENCE)[0][0].tolist()) == {4, 6, 0, 3}
    assert set(o.search(q, 4, 4, mode=O.CANONICAL)[0][0].tolist()) == {4, 6, 0, 2}
    for ef in range(1, 9):
        for k in range(1, ef + 1):
            want = o.search(q, k, ef, mode=O.REFERENCE)
            got = g.knn_query_traced(q, k, ef=ef, tie_order="reference")
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (ef, k)


@pytest.mark.parametrize("M", [6, 16, 24])  # 12 and 32 links in one unit, 48 in two
@pytest.mark.parametrize("values,dim", [(8, 16), (30, 16), (12, 8)])
def test_small_integers_against_replay(tmp_path, M, values, dim):
    rng = np.random.default_rng(M * 100 + values)
    x = rng.integers(0, values, (1200, dim)).astype(np.float32)
    write_graph(tmp_path / "g.bin", x, "l2", M, seed=M)
    g = H.Index("l2", dim)
    g.load_index(str(tmp_path / "g.bin"))
    for _ in range(6):
        q = rng.integers(0, values, (20000, dim)).astype(np.float32)
        for ef, k in ((10, 10), (4, 4), (16, 5)):
            got = g.knn_query_traced(q, k, ef=ef, tie_order="reference")
            want = g.knn_query_traced(q, k, ef=ef, tie_order="replay")
            for a, b in zip(got[:3], want[:3]):
                assert np.array_equal(a, b)
            assert np.array_equal(got[3][:, 2], want[3][:, 2])  # expansions
