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


@pytest.mark.parametrize("prec", ["bf16", "fp8"])
@pytest.mark.parametrize("space", ["l2", "ip"])
@pytest.mark.parametrize("dim", [2, 5, 16, 20, 33, 100, 129])
def test_rerank_forms(prec, space, dim):
    """Every row re-ranked: the low-precision scan is the exact one."""
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((1000, dim)).astype(np.float32)
    q = rng.standard_normal((130, dim)).astype(np.float32)
    g = H.BFIndex(space, dim)
    g.init_index(1000)
    g.add_items(x, rng.permutation(1000))
    el, ed = g.knn_query(q, k=10)
    l, d, c, _ = g.knn_query_traced(q, 10, precision=prec, rerank=1000)
    assert np.array_equal(l, el) and np.array_equal(d.view(np.uint32), ed.view(np.uint32))


@pytest.mark.parametrize("prec", ["bf16", "fp8"])
def test_lists_that_overflow(prec):
    """Queries whose candidate list overflows are answered exactly: many tied
    rows under the threshold, and a sample without any admissible row."""
    rng = np.random.default_rng(7)
    x = rng.integers(0, 2, (60000, 16)).astype(np.float32)
    x[::2] = 1.0
    q = rng.integers(0, 2, (300, 16)).astype(np.float32)
    g = H.BFIndex("l2", 16)
    g.init_index(60000)
    g.add_items(x)
    for filt in (None, lambda v: v % 12 != 0 and v % 15 != 0):
        g.precision = "fp32"
        el, ed = g.knn_query(q, k=10, filter=filt)
        g.precision = prec
        l, d = g.knn_query(q, k=10, filter=filt)
        lt, dt, _, tr = g.knn_query_traced(q, 10, filter=filt, precision=prec)
        assert np.array_equal(l, lt) and np.array_equal(d, dt)
        redo = tr[:, 2] == 1
        assert redo.any()
        assert np.array_equal(l[redo], el[redo]) and np.array_equal(d[redo], ed[redo])


def _clusters(rng, n, dim, sigma):
    c = rng.standard_normal((max(4, n // 500), dim)).astype(np.float32)
    return (c[rng.integers(0, len(c), n)] + sigma * rng.standard_normal((n, dim))).astype(np.float32)


@pytest.mark.parametrize("space", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("dim", [33, 100, 128])
@pytest.mark.parametrize("sigma", [0.02, 0.5, 30.0])
def test_certified_scan(tmp_path, space, dim, sigma):
    """Batches large enough for the tensor-core route of the exact scan: tight
    clusters (distances far below the scores' error), loose ones, and rows
    whose norms differ; k on both sides of its sample sizes; a mask."""
    rng = np.random.default_rng(dim)
    x = _clusters(rng, 20000, dim, sigma)
    x[::1000] *= 20.0
    g, o = _pair(tmp_path, x, space)
    q = _clusters(rng, 700, dim, sigma)
    q[::2] = x[rng.integers(0, 20000, 350)] + np.float32(0.01)
    for k in (1, 100, 101, 256):
        _same(g, o, q, k)
    _same(g, o, q, 10, filt=lambda v: v % 127 != 0 and v % 3 == 0)
    _same(g, o, q, 10, filt=lambda v: v % 2000 == 5)


def test_certified_scan_ties_and_range(tmp_path):
    rng = np.random.default_rng(11)
    x = rng.integers(0, 2, (30000, 40)).astype(np.float32)
    x[10000:] = x[:20000]  # every distance at least twice
    g, o = _pair(tmp_path, x, "l2")
    q = rng.integers(0, 2, (600, 40)).astype(np.float32)
    _same(g, o, q, 10)
    for scale in (1e-21, 3e18):  # squares under- and overflow float32
        g, o = _pair(tmp_path, x * np.float32(scale), "l2")
        _same(g, o, q * np.float32(scale), 10)
