"""Exact scan over the forms its kernels branch on (needs a B200): every
summation form of the distances, row / query / group tile edges, ties beyond
the selection's capacity, k beyond its group bound, masks, query batches.
Bit-identical to BruteforceSearch::searchKnn throughout."""
import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import pickling
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _pair(tmp_path, x, space):
    rows = pickling.normalize_rows(x) if space == "cosine" else x
    (tmp_path / "bf.bin").write_bytes(
        pickling.bf_rows_to_file(rows, np.arange(len(x), dtype=np.uint64), len(x), x.shape[1]))
    g = H.BFIndex(space, x.shape[1])
    g.load_index(str(tmp_path / "bf.bin"))
    return g, O.Bf(str(tmp_path / "bf.bin"), space, x.shape[1])


def _same(g, o, q, k, filt=None):
    n = g.get_current_count()
    gl, gd, gc, _ = g.knn_query_traced(q, k, filter=filt)
    allow = None if filt is None else np.array([filt(i) for i in range(n)], np.uint8)
    ol, od, oc = o.search(q, k, allow=allow)
    assert np.array_equal(gc, oc)
    for i in range(q.shape[0]):
        c = int(oc[i])
        assert np.array_equal(gl[i, :c], ol[i, :c])
        assert np.array_equal(gd[i, :c].view(np.uint32), od[i, :c].view(np.uint32))


@pytest.mark.parametrize("space", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("dim", [1, 3, 4, 5, 15, 16, 17, 20, 31, 32, 36, 47, 48, 100, 129])
def test_forms_and_query_tiles(tmp_path, space, dim):
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((777, dim)).astype(np.float32)
    g, o = _pair(tmp_path, x, space)
    for nq in (1, 2, 5, 9):
        _same(g, o, rng.standard_normal((nq, dim)).astype(np.float32), 7)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1025, 20000])
def test_row_edges_and_k(tmp_path, n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 24)).astype(np.float32)
    g, o = _pair(tmp_path, x, "l2")
    q = rng.standard_normal((3, 24)).astype(np.float32)
    for k in (1, 10, 512, 513, 1500):
        _same(g, o, q, k)
        _same(g, o, q, k, filt=lambda v: v % 7 == 3)


def test_ties_beyond_the_selection(tmp_path):
    rng = np.random.default_rng(1)
    x = rng.integers(0, 2, (30000, 8)).astype(np.float32)  # 256 distinct rows
    g, o = _pair(tmp_path, x, "l2")
    q = rng.integers(0, 2, (5, 8)).astype(np.float32)
    for k in (1, 50, 1000):
        _same(g, o, q, k)
    same = np.ones((5000, 8), np.float32)
    g, o = _pair(tmp_path, same, "ip")
    _same(g, o, q, 20)


def test_query_batches(tmp_path):
    """More distance keys than one batch holds."""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((70000, 4)).astype(np.float32)
    g, o = _pair(tmp_path, x, "cosine")
    _same(g, o, rng.standard_normal((1001, 4)).astype(np.float32), 10)
