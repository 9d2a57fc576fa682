"""Performance cases of the query path, through the package's public calls.

Three families, all called the way a user's program calls them (host arrays in,
host arrays out):

``graph``  ``Index.knn_query`` on an HNSW index: the graph is built here on the
           GPU (nearest-neighbour lists pruned by the HNSW diversity rule, linked
           in both directions, with the usual geometric upper levels) and handed
           over as a pickled index state, as a program with a saved index does;
``scan``   ``BFIndex.knn_query``: exhaustive search in float32 (the exact scan)
           or over the bf16 / fp8 copies;
``train``  ``learned.train``: the network of the learned early stop.

Data follow the distributions of ``hnsw_rabitq_b200.datasets``: "u255" integer
valued Gaussian mixtures in [0, 255], "unit" unit vectors around unit centres,
"sigma" mixtures whose components differ in spread, "uniform" U[0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hnsw_rabitq_b200 import BFIndex, Index, learned

DEV = "cuda"


def listed():
    return [
        # one interactive query against a small index: the latency of a call
        dict(name="graph_one_query", kind="graph", data="u255", n=100_000, dim=128, space="l2", M=16, nq=1, k=10,
             ef=50, tie="reference", precision="fp32", deleted=0.0, filtered=False),
        # the headline workload in the default settings (the reference's order)
        dict(name="graph_1m_default", kind="graph", data="u255", n=1_000_000, dim=128, space="l2", M=16, nq=10_000,
             k=10, ef=50, tie="reference", precision="fp32", deleted=0.0, filtered=False),
        # word-vector like: a dimension that is no multiple of 16, cosine
        dict(name="graph_cosine_100", kind="graph", data="sigma", n=200_000, dim=100, space="cosine", M=16, nq=1000,
             k=10, ef=100, tie="reference", precision="fp32", deleted=0.0, filtered=False),
        # the fast approximate form: fp8 traversal with float32 re-rank
        dict(name="graph_fp8", kind="graph", data="u255", n=500_000, dim=128, space="l2", M=16, nq=10_000, k=10,
             ef=52, tie="id", precision="fp8", deleted=0.0, filtered=False),
        # wide graph of a hard mixture, the id order
        dict(name="graph_m32_96", kind="graph", data="sigma", n=250_000, dim=96, space="l2", M=32, nq=2000, k=10,
             ef=64, tie="id", precision="fp32", deleted=0.0, filtered=False),
        # embeddings with deleted elements and a filter, many results
        dict(name="graph_filtered_768", kind="graph", data="unit", n=100_000, dim=768, space="ip", M=16, nq=100,
             k=100, ef=256, tie="id", precision="fp32", deleted=0.05, filtered=True),
        # one exact query of a ragged dimension: a small scan
        dict(name="scan_one_query", kind="scan", data="sigma", n=100_000, dim=100, space="cosine", nq=1, k=10,
             precision="fp32", filtered=False),
        # ground truth of a small uniform set
        dict(name="scan_uniform_10k", kind="scan", data="uniform", n=10_000, dim=128, space="l2", nq=1000, k=10,
             precision="fp32", filtered=False),
        # exact search over embeddings
        dict(name="scan_embed_768", kind="scan", data="unit", n=200_000, dim=768, space="ip", nq=500, k=100,
             precision="fp32", filtered=False),
        # tensor-core scan of embeddings, a large batch
        dict(name="scan_bf16_768", kind="scan", data="unit", n=200_000, dim=768, space="ip", nq=5000, k=100,
             precision="bf16", filtered=False),
        # fp8 scan of byte-like vectors with a filter
        dict(name="scan_fp8_128", kind="scan", data="u255", n=300_000, dim=128, space="l2", nq=2000, k=10,
             precision="fp8", filtered=True),
        # training the early-stop network on recorded checkpoints
        dict(name="train_stop", kind="train", n=60_000, epochs=4, batch=1024),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["graph", "scan", "train"], [6, 5, 1])[0]
    if kind == "train":
        return dict(kind="train", n=_logint(rng, 2000, 60_000), epochs=rng.randint(1, 4),
                    batch=rng.choice([256, 500, 1024, 2048]))
    data = rng.choice(["u255", "sigma", "unit"])
    space = {"u255": "l2", "sigma": rng.choice(["l2", "cosine"]), "unit": rng.choice(["ip", "cosine"])}[data]
    if kind == "graph":
        precision = rng.choices(["fp32", "bf16", "fp8"], [6, 1, 2])[0]
        dim = _logint(rng, 24, 768)
        if precision != "fp32" or rng.random() < 0.5:
            dim = max(32, dim // 32 * 32)
        if precision == "fp8" and dim > 128:
            dim = dim // 128 * 128
        M = rng.choice([8, 16, 16, 32]) if precision == "fp32" else 16
        special = precision != "fp8" and rng.random() < 0.25
        k = rng.choice([1, 10, 10, 100])
        ef = max(k, _logint(rng, 24, 300))
        return dict(kind="graph", data=data, n=min(_logint(rng, 20_000, 400_000), 40_000_000 // dim), dim=dim,
                    space=space, M=M, nq=min(_logint(rng, 1, 10_000), 50_000_000 // (dim * ef)), k=k, ef=ef,
                    tie="id" if precision != "fp32" else rng.choice(["reference", "reference", "id"]),
                    precision=precision, deleted=0.05 if special else 0.0, filtered=special and rng.random() < 0.5)
    precision = rng.choices(["fp32", "bf16", "fp8"], [3, 1, 1])[0]
    dim = _logint(rng, 24, 768)
    if precision != "fp32" or rng.random() < 0.5:
        dim = max(32, dim // 32 * 32)
    n = min(_logint(rng, 5000, 400_000), 150_000_000 // dim)
    return dict(kind="scan", data=data, n=n, dim=dim, space=space,
                nq=_logint(rng, 1, 500 if precision == "fp32" else 5000), k=rng.choice([1, 10, 10, 100]),
                precision=precision, filtered=rng.random() < 0.25)


# ------------------------------------------------------------------ vectors
def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + stream)
    return g


def _unit(x):
    return x / x.norm(dim=1, keepdim=True).clamp_min(1e-20)


def _vectors(case, seed):
    """(base rows, query rows) on the GPU, float32."""
    n, dim, nq = case["n"], case["dim"], case["nq"]
    data = case["data"]
    if data == "uniform":
        return (torch.rand(n, dim, generator=_gen(seed, 0), device=DEV),
                torch.rand(nq, dim, generator=_gen(seed, 1), device=DEV))
    comps = max(16, n // 1000) if data != "unit" else max(16, min(256, n // 400))
    gc = _gen(seed, 7)
    if data == "u255":
        centres = torch.rand(comps, dim, generator=gc, device=DEV) * 255.0
        sigma = torch.full((comps, 1), 20.0, device=DEV)
    elif data == "sigma":
        centres = torch.randn(comps, dim, generator=gc, device=DEV)
        sigma = torch.exp(torch.empty(comps, 1, device=DEV).uniform_(math.log(0.05), math.log(0.5), generator=gc))
    else:
        centres = _unit(torch.randn(comps, dim, generator=gc, device=DEV))
        sigma = torch.full((comps, 1), 0.3 / math.sqrt(dim), device=DEV)

    def rows(m, g):
        c = torch.randint(0, comps, (m,), generator=g, device=DEV)
        v = centres[c] + torch.randn(m, dim, generator=g, device=DEV) * sigma[c]
        if data == "u255":
            return v.round_().clamp_(0.0, 255.0)
        return _unit(v) if data == "unit" else v

    return rows(n, _gen(seed, 0)), rows(nq, _gen(seed, 1))


# ------------------------------------------------------------- graph building
def _neighbours(x, cand, gen):
    """Close rows of every row (ids int64 [n, cand], -1: none): exact for small sets,
    else by balanced random splits of the set into leaves, three times over."""
    n = x.shape[0]
    if n <= 1:
        return torch.full((n, cand), -1, dtype=torch.int64, device=DEV)
    sq = x.square().sum(1)
    if n <= 32768:
        kk = min(cand, n - 1)
        out = torch.empty(n, kk, dtype=torch.int64, device=DEV)
        for s in range(0, n, 4096):
            e = min(n, s + 4096)
            d = sq[None, :] - 2.0 * (x[s:e] @ x.t())
            d[torch.arange(e - s, device=DEV), torch.arange(s, e, device=DEV)] = float("inf")
            out[s:e] = d.topk(kk, dim=1, largest=False).indices
        if kk < cand:
            out = torch.cat([out, out.new_full((n, cand - kk), -1)], 1)
        return out
    depth = max(1, round(math.log2(n / 4096)))
    leaves = 1 << depth
    size = -(-n // leaves)
    total = leaves * size
    per = max(8, cand // 2)
    found = []
    for _ in range(3):
        # repeats of random rows (numbers from n on) even out the leaves
        order = torch.cat([torch.randperm(n, generator=gen, device=DEV),
                           torch.randint(n, 2 * n, (total - n,), generator=gen, device=DEV)])
        parts = 1
        for _ in range(depth):
            order = order.view(parts, -1)
            m = order.shape[1]
            a = x[order[:, torch.randint(0, m, (1,), generator=gen, device=DEV)].view(-1) % n]
            b = x[order[:, torch.randint(0, m, (1,), generator=gen, device=DEV)].view(-1) % n]
            direction = a - b
            key = torch.empty(parts, m, device=DEV)
            step = max(1, (1 << 28) // (m * x.shape[1]))
            for s in range(0, parts, step):
                e = min(parts, s + step)
                if m * x.shape[1] > 1 << 29:  # one part at a time: no gathered copy
                    key[s:e] = (x @ direction[s])[order[s] % n].view(1, -1)
                else:
                    key[s:e] = torch.bmm(x[order[s:e] % n], direction[s:e, :, None]).squeeze(2)
            order = order.gather(1, key.argsort(dim=1, stable=True))
            parts *= 2
            order = order.reshape(parts, m // 2)
        ids = torch.full((n, per), -1, dtype=torch.int64, device=DEV)
        step = max(1, (1 << 28) // (size * max(size, x.shape[1])))
        for s in range(0, leaves, step):
            own = order[s:s + step].reshape(-1) < n
            o = order[s:s + step] % n
            xl = x[o]
            d = sq[o][:, None, :] - 2.0 * torch.bmm(xl, xl.transpose(1, 2))
            d.masked_fill_(o[:, None, :] == o[:, :, None], float("inf"))
            near = d.topk(per, dim=2, largest=False).indices
            got = o[:, None, :].expand(-1, size, -1).gather(2, near).reshape(-1, per)
            ids[o.reshape(-1)[own]] = got[own]
        found.append(ids)
    return torch.cat(found, 1)


def _links(x, cand_ids, M, cap, gen):
    """Links of every row: candidates pruned by the HNSW diversity rule, some long
    links (the closest of 32 random rows each: an incrementally built graph has such
    links from its first insertions), then linked back, at most cap a row (int32 [n, cap], -1: unused)."""
    n, C = cand_ids.shape
    keep = torch.full((n, M), -1, dtype=torch.int64, device=DEV)
    kd = torch.full((n, M), float("inf"), device=DEV)
    far = M // 4 if n > 1024 else 0
    near = M - far
    if far:
        block = max(1, (1 << 27) // (32 * far * x.shape[1]))
        for s in range(0, n, block):
            v = x[s:s + block]
            ids = torch.randint(0, n - 1, (v.shape[0], far * 32), generator=gen, device=DEV)
            ids += ids >= torch.arange(s, s + v.shape[0], device=DEV)[:, None]
            d = (x[ids] - v[:, None, :]).square().sum(2).view(-1, far, 32)
            d, at = d.min(2)
            keep[s:s + block, near:] = ids.view(-1, far, 32).gather(2, at[:, :, None]).squeeze(2)
            kd[s:s + block, near:] = d
    width = min(C, 2 * M + 8)
    step = max(1, (1 << 27) // (C * x.shape[1]))
    inf = float("inf")
    for s in range(0, n, step):
        e = min(n, s + step)
        ids = cand_ids[s:e].sort(dim=1).values
        bad = ids < 0
        bad[:, 1:] |= ids[:, 1:] == ids[:, :-1]
        safe = ids.clamp_min(0)
        d = (x[safe] - x[s:e, None, :]).square().sum(2).masked_fill_(bad, inf)
        d, at = d.topk(width, dim=1, largest=False)
        ids = safe.gather(1, at)
        v = x[ids]
        vv = v.square().sum(2)
        pair = vv[:, :, None] + vv[:, None, :] - 2.0 * torch.bmm(v, v.transpose(1, 2))
        chosen = torch.zeros(e - s, width, dtype=torch.bool, device=DEV)
        count = torch.zeros(e - s, dtype=torch.int64, device=DEV)
        for j in range(width):
            closest = torch.where(chosen, pair[:, j], inf).amin(1)
            ok = (d[:, j] < closest) & (count < near) & (d[:, j] < inf)
            chosen[:, j] = ok
            count += ok
        rank = chosen.cumsum(1) - 1
        rr, cc = chosen.nonzero(as_tuple=True)
        keep[s + rr, rank[rr, cc]] = ids[rr, cc]
        kd[s + rr, rank[rr, cc]] = d[rr, cc]
    # both directions, without repeats, closest first
    src = torch.arange(n, device=DEV)[:, None].expand(n, M)[keep >= 0]
    dst, dist = keep[keep >= 0], kd[keep >= 0]
    a, b, w = torch.cat([src, dst]), torch.cat([dst, src]), torch.cat([dist, dist])
    code, first = (a * n + b).sort(stable=True)
    uniq = torch.ones_like(code, dtype=torch.bool)
    uniq[1:] = code[1:] != code[:-1]
    first = first[uniq]
    a, b, w = a[first], b[first], w[first]
    order = w.sort(stable=True).indices
    a, b = a[order], b[order]
    order = a.sort(stable=True).indices
    a, b = a[order], b[order]
    start = torch.searchsorted(a, torch.arange(n, device=DEV))
    rank = torch.arange(a.shape[0], device=DEV) - start[a]
    out = torch.full((n, cap), -1, dtype=torch.int32, device=DEV)
    ok = rank < cap
    out[a[ok], rank[ok]] = b[ok].to(torch.int32)
    return out


def _state(case, x, seed):
    """The pickled state (hnswlib's getIndexParams dict) of a graph over rows x."""
    n, dim = x.shape
    M = case["M"]
    M0 = 2 * M
    gen = _gen(seed, 3)
    u = torch.rand(n, generator=gen, device=DEV).clamp_min(1e-12)
    levels = (-torch.log(u) / math.log(M)).floor().to(torch.int64)
    top = int(levels.max())
    sums = torch.zeros(n, dtype=torch.int64, device=DEV)
    if n > 1:
        sums[1:] = levels.cumsum(0)[:-1]
    rows = int(levels.sum())
    upper = torch.zeros(max(rows, 1), 1 + M, dtype=torch.int32, device=DEV)
    for level in range(1, top + 1):
        members = (levels >= level).nonzero().view(-1)
        m = members.shape[0]
        links = _links(x[members], _neighbours(x[members], 2 * M + 8, gen), M, M, gen)
        have = links >= 0
        at = sums[members] + level - 1
        upper[at, 0] = have.sum(1).to(torch.int32)
        ids = members[links.clamp_min(0).to(torch.int64)].to(torch.int32)
        upper[at, 1:] = torch.where(have, ids, 0) if m > 1 else 0
    links = _links(x, _neighbours(x, 2 * M + 8, gen), M, M0, gen)
    have = links >= 0
    rec = torch.zeros(n, 1 + M0 + dim + 2, dtype=torch.int32, device=DEV)
    rec[:, 0] = have.sum(1).to(torch.int32)
    if case["deleted"]:
        rec[:, 0] |= (torch.rand(n, generator=gen, device=DEV) < case["deleted"]).to(torch.int32) << 16
    rec[:, 1:1 + M0] = torch.where(have, links, 0)
    rec[:, 1 + M0:1 + M0 + dim] = x.view(torch.int32)
    rec[:, -2] = torch.arange(n, device=DEV, dtype=torch.int32)
    size_data = rec.shape[1] * 4
    return dict(ser_version=1, space=case["space"], dim=dim, index_inited=True, ep_added=True,
                normalize=case["space"] == "cosine", num_threads=-1, seed=100, offset_level0=0, max_elements=n,
                cur_element_count=n, size_data_per_element=size_data, label_offset=size_data - 8,
                offset_data=4 + 4 * M0, max_level=top, enterpoint_node=int(levels.argmax()), max_M=M, max_M0=M0, M=M,
                mult=1.0 / math.log(M), ef_construction=200, ef=case["ef"],
                has_deletions=bool(case["deleted"]), size_links_per_element=4 + 4 * M,
                allow_replace_deleted=False, element_levels=levels.cpu().numpy().astype(np.int32),
                data_level0=rec.cpu().numpy().view(np.int8).reshape(-1),
                link_lists=upper[:rows].cpu().numpy().view(np.int8).reshape(-1))


# ------------------------------------------------------------------ the cases
def _keep(label):
    """The filter of the filtered cases: two labels of three."""
    return label % 3 != 0


def prepare(case, seed):
    if case["kind"] == "train":
        rng = np.random.default_rng(seed)
        feats = rng.normal(size=(case["n"], learned.F)).astype(np.float32)
        feats = feats * rng.uniform(0.2, 4.0, learned.F).astype(np.float32) + rng.normal(size=learned.F).astype(np.float32)
        score = feats @ rng.normal(size=learned.F) + rng.normal(size=case["n"])
        labels = (score > np.quantile(score, 0.4)).astype(np.float32)
        return dict(case=case, feats=feats, labels=labels, params=learned.init_params(feats, seed), seed=int(seed))
    x, q = _vectors(case, seed)
    state = dict(case=case, queries=q.cpu().numpy())
    if case["kind"] == "graph":
        if case["space"] == "cosine":
            x = _unit(x)
        index = Index.from_params(_state(case, x, seed))
        index.tie_order = case["tie"]
        index.precision = case["precision"]
        if case["filtered"]:
            state["filter"] = index.register_filter(_keep)
    else:
        index = BFIndex(case["space"], case["dim"])
        index.init_index(case["n"])
        index.add_items(x.cpu().numpy())
        index.precision = case["precision"]
        # the index goes to the GPU at its first query
        index.knn_query(state["queries"][:1], k=1)
        if case["filtered"]:
            state["filter"] = index.register_filter(_keep)
    state["index"] = index
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        return learned.train(state["feats"], state["labels"], params=state["params"], epochs=case["epochs"],
                             batch=case["batch"], seed=state["seed"])
    return state["index"].knn_query(state["queries"], k=case["k"], filter=state.get("filter"))


def work(case):
    if case["kind"] == "train":
        n, e, h, f = case["n"], case["epochs"], learned.H, learned.F
        return dict(bytes=n * (f + 1) * 4 + 2 * 4 * learned.N_PARAMS, flops=6.0 * n * e * (f * h + h * h + h))
    n, dim, nq, k = case["n"], case["dim"], case["nq"], case["k"]
    io = nq * dim * 4 + nq * k * 12 + nq * 4
    element = {"fp32": 4, "bf16": 2, "fp8": 1}[case["precision"]]
    if case["kind"] == "scan":
        return dict(bytes=io + n * dim * element, flops=2.0 * nq * n * dim)
    # about ef expansions a query, each with one link list and M rows not seen before
    row = dim * element
    walk = nq * case["ef"] * (8 * case["M"] + case["M"] * row)
    return dict(bytes=io + min(walk, n * (8 * case["M"] + row)) if nq < 100 else io + walk,
                flops=2.0 * nq * case["ef"] * case["M"] * dim)


def exact(case, seed):
    """The exact nearest neighbours' distances in 64 bits: what a scan returns, and
    what a graph search approximates.  Labels are whole numbers; deleted or
    filtered elements leave a graph search no simple exact form here."""
    if case["kind"] == "train" or (case["kind"] == "graph" and (case["deleted"] or case["filtered"])):
        return None
    x, q = _vectors(case, seed)
    x, q = x.double(), q.double()
    if case["space"] == "cosine":
        x, q = _unit(x), _unit(q)
    sq = x.square().sum(1)
    allowed = None
    if case["filtered"]:
        allowed = torch.arange(case["n"], device=DEV) % 3 != 0
    out = np.empty((case["nq"], case["k"]), np.float64)
    step = max(1, (1 << 28) // case["n"])
    for s in range(0, case["nq"], step):
        b = q[s:s + step]
        dot = b @ x.t()
        d = sq[None, :] + b.square().sum(1)[:, None] - 2.0 * dot if case["space"] == "l2" else 1.0 - dot
        if allowed is not None:
            d = d.masked_fill(~allowed, float("inf"))
        out[s:s + step] = d.topk(case["k"], dim=1, largest=False, sorted=True).values.cpu().numpy()
    return None, out
