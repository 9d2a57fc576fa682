"""Graph search over the forms its beam branches on (needs a B200): summation
forms of the distances, lists of up to 32, 64 and more links, staging batches,
and distance ties that steer the reference's heaps (lazy heaps) -- against the
oracle's reference and canonical runs, bit for bit.  The graphs are built here
(nearest neighbours and random links, geometric levels)."""
import numpy as np
import pytest

import hnsw_rabitq_b200 as H
from hnsw_rabitq_b200 import pickling
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def write_graph(path, x, space, M, seed=0, deleted=0.0):
    rng = np.random.default_rng(seed)
    n, dim = x.shape
    rows = pickling.normalize_rows(x) if space == "cosine" else x.astype(np.float32)
    levels = np.floor(-np.log(rng.random(n) + 1e-12) / np.log(M)).astype(np.int32)
    top = int(levels.max())

    def links(members, cap):
        v = rows[members].astype(np.float64)
        d = (v * v).sum(1)[None] - 2 * v @ v.T
        np.fill_diagonal(d, np.inf)
        out = []
        for i in range(len(members)):
            near = np.argsort(d[i], kind="stable")[: max(1, cap * 2 // 3)]
            far = rng.integers(0, len(members), cap // 3 + 1)
            ids = [int(j) for j in dict.fromkeys(np.concatenate([near, far]).tolist()) if j != i and len(members) > 1]
            rng.shuffle(ids)
            out.append([int(members[j]) for j in ids[: rng.integers(max(1, cap // 2), cap + 1)]])
        return out

    M0 = 2 * M
    size = 4 + 4 * M0 + 4 * dim + 8
    rec = np.zeros((n, size), np.uint8)
    for i, l in enumerate(links(np.arange(n), M0)):
        head = np.zeros(1 + M0, np.uint32)
        head[0] = len(l) | (int(rng.random() < deleted) << 16)
        head[1:1 + len(l)] = l
        rec[i, :4 + 4 * M0] = head.view(np.uint8)
    rec[:, 4 + 4 * M0:-8] = rows.view(np.uint8).reshape(n, -1)
    labels = (rng.permutation(n) + 7).astype(np.uint64)
    rec[:, -8:] = labels.view(np.uint8).reshape(n, 8)
    upper = {}
    for level in range(1, top + 1):
        members = np.nonzero(levels >= level)[0]
        for i, l in zip(members, links(members, M)):
            row = np.zeros(1 + M, np.uint32)
            row[0] = len(l)
            row[1:1 + len(l)] = l
            upper.setdefault(int(i), []).append(row)
    flat = [r for i in range(n) for r in upper.get(i, [])]
    state = dict(offset_level0=0, max_elements=n, cur_element_count=n, size_data_per_element=size,
                 label_offset=size - 8, offset_data=4 + 4 * M0, max_level=top, enterpoint_node=int(levels.argmax()),
                 max_M=M, max_M0=M0, M=M, mult=1 / np.log(M), ef_construction=100, size_links_per_element=4 + 4 * M,
                 element_levels=levels, data_level0=rec.reshape(-1),
                 link_lists=np.concatenate(flat).view(np.uint8) if flat else np.zeros(0, np.uint8))
    path.write_bytes(pickling.state_to_file_bytes(state))
    return labels


def _same(got, want, trace=True):
    l, d, c, t = got
    ol, od, oc, ot = want
    assert np.array_equal(c, oc)
    for i in range(len(c)):
        k = int(c[i])
        assert np.array_equal(l[i, :k], ol[i, :k]), i
        assert np.array_equal(d[i, :k].view(np.uint32), od[i, :k].view(np.uint32)), i
    if trace:
        assert np.array_equal(t[:, 2], ot[:, 2])  # level-0 expansions


def _check(tmp_path, x, q, space, M, shapes, deleted=0.0, filt=None):
    labels = write_graph(tmp_path / "g.bin", x, space, M, seed=M, deleted=deleted)
    o = O.Hnsw(str(tmp_path / "g.bin"), space, x.shape[1])
    g = H.Index(space, x.shape[1])
    g.load_index(str(tmp_path / "g.bin"))
    allow = None if filt is None else np.array([filt(int(v)) for v in labels], np.uint8)
    for ef, k in shapes:
        for mode, order in ((O.REFERENCE, "reference"), (O.REFERENCE, "replay"), (O.CANONICAL, "id")):
            want = o.search(q, k, max(ef, k), mode=mode, allow=allow, trace=True)
            for nq in (len(q), 3):
                _same(g.knn_query_traced(q[:nq], k, ef=ef, tie_order=order, filter=filt),
                      tuple(w[:nq] for w in want))
        assert g.get_status() == 0


@pytest.mark.parametrize("space", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("dim", [3, 7, 16, 20, 33, 48, 100, 160])
def test_dims(tmp_path, space, dim):
    rng = np.random.default_rng(dim)
    x = rng.standard_normal((1500, dim)).astype(np.float32)
    q = rng.standard_normal((150, dim)).astype(np.float32)
    _check(tmp_path, x, q, space, 16, [(1, 1), (20, 10), (90, 33)])


@pytest.mark.parametrize("M", [2, 8, 17, 32, 40])
def test_list_lengths(tmp_path, M):
    rng = np.random.default_rng(M)
    x = rng.standard_normal((1200, 24)).astype(np.float32)
    q = rng.standard_normal((120, 24)).astype(np.float32)
    _check(tmp_path, x, q, "l2", M, [(10, 10), (64, 5)])


@pytest.mark.parametrize("M", [8, 16, 32])
@pytest.mark.parametrize("values,dim", [(2, 16), (3, 12), (4, 33), (6, 64)])
def test_ties(tmp_path, M, values, dim):
    """Small integers: ties at the next candidate, at the pool's edge and
    across the k-th result, up to searches that log more than fits."""
    rng = np.random.default_rng(values)
    x = rng.integers(0, values, (1500, dim)).astype(np.float32)
    q = rng.integers(0, values, (200, dim)).astype(np.float32)
    _check(tmp_path, x, q, "l2", M, [(1, 1), (4, 2), (16, 10), (50, 10), (150, 100)])


@pytest.mark.parametrize("dim,M", [(16, 16), (20, 16), (128, 32), (33, 32)])
@pytest.mark.parametrize("deleted,filt", [(0.3, None), (0.0, 3), (0.2, 2)])
def test_deleted_and_filtered(tmp_path, dim, M, deleted, filt):
    rng = np.random.default_rng(dim)
    x = rng.integers(0, 9, (1500, dim)).astype(np.float32)
    q = rng.integers(0, 9, (100, dim)).astype(np.float32)
    _check(tmp_path, x, q, "l2", M, [(10, 5), (60, 20)], deleted=deleted,
           filt=None if filt is None else (lambda v: v % filt == 0))


def test_wide_rows(tmp_path):
    """Rows of which only a few fit a staging batch."""
    rng = np.random.default_rng(0)
    x = rng.standard_normal((600, 1024)).astype(np.float32)
    q = rng.standard_normal((400, 1024)).astype(np.float32)
    _check(tmp_path, x, q, "ip", 16, [(40, 10)])


@pytest.mark.parametrize("M", [16, 32])
@pytest.mark.parametrize("values,dim,n", [(16, 16, 4000), (40, 12, 4000), (256, 8, 4000), (256, 32, 3000)])
def test_occasional_ties(tmp_path, M, values, dim, n):
    """Ties that mostly cannot change the result: most queries run without
    heaps, and the rest must be recognised."""
    rng = np.random.default_rng(values)
    x = rng.integers(0, values, (n, dim)).astype(np.float32)
    q = rng.integers(0, values, (1500, dim)).astype(np.float32)
    _check(tmp_path, x, q, "l2", M, [(10, 10), (24, 5), (60, 10)])
