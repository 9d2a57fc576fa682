"""The rule by which the tie-exact beam keeps the id-order run's result: a
query whose run met no tie that can matter has the reference's result.  Both
runs are simulated on random graphs with small integer distances (CPU): the
reference's two heaps in libstdc++'s layout, and the (distance, id) order with
the rule's bookkeeping, expansion by expansion as the kernel does it."""
import random

import pytest


def push(h, v, less):
    h.append(v)
    i = len(h) - 1
    while i > 0:
        p = (i - 1) // 2
        if not less(h[p], v):
            break
        h[i] = h[p]
        i = p
    h[i] = v


def pop(h, less):
    top = h[0]
    v = h.pop()
    n = len(h)
    if n:
        i = c = 0
        while c < (n - 1) // 2:
            c = 2 * (c + 1)
            if less(h[c], h[c - 1]):
                c -= 1
            h[i] = h[c]
            i = c
        if n % 2 == 0 and c == (n - 2) // 2:
            c = 2 * (c + 1)
            h[i] = h[c - 1]
            i = c - 1
        while i > 0:
            p = (i - 1) // 2
            if not less(h[p], v):
                break
            h[i] = h[p]
            i = p
        h[i] = v
    return top


def far(a, b):  # top_candidates: the largest distance on top
    return a[0] < b[0]


def near(a, b):  # candidate_set: the smallest distance on top
    return a[0] > b[0]


def reference(links, dist, ep, ef, k):
    top, cand, seen, expanded = [], [], {ep}, 0
    push(top, (dist[ep], ep), far)
    push(cand, (dist[ep], ep), near)
    lb = dist[ep]
    while cand:
        if cand[0][0] > lb:
            break
        _, c = pop(cand, near)
        expanded += 1
        for x in links[c]:
            if x in seen:
                continue
            seen.add(x)
            if len(top) < ef or lb > dist[x]:
                push(cand, (dist[x], x), near)
                push(top, (dist[x], x), far)
                if len(top) > ef:
                    pop(top, far)
                lb = top[0][0]
    while len(top) > k:
        pop(top, far)
    return sorted(top), expanded


def id_order(links, dist, ep, ef, k):
    """(result, expansions, whether a tie can matter)."""
    pool, done, seen, expanded = [(dist[ep], ep)], {ep}, {ep}, 1
    node, tie_a, tie_b = ep, None, None
    while True:
        # the reference's sequential test; lowerBound at the start of the expansion
        lbk = pool[-1][0] if len(pool) == ef else None
        fresh = [x for x in links[node] if x not in seen]
        seen.update(fresh)
        if tie_a is not None and lbk is not None and any(dist[x] == lbk for x in fresh):
            return None, None, True
        live = [x for x in fresh if lbk is None or dist[x] < lbk]
        accepted = [x for i, x in enumerate(live)
                    if sum(p[0] <= dist[x] for p in pool) + sum(dist[y] <= dist[x] for y in live[:i]) < ef]
        waiting = [p for p in pool if p[1] not in done] + [(dist[x], x) for x in accepted]
        nxt = min(waiting) if waiting else None
        if nxt and sum(w[0] == nxt[0] for w in waiting) > 1:
            tie_a = nxt[0] if tie_a is None else max(tie_a, nxt[0])
        pool = sorted(pool + [(dist[x], x) for x in accepted])
        if len(pool) > ef:
            if pool[ef][0] == pool[ef - 1][0]:
                tie_b = pool[ef][0]
            pool = pool[:ef]
        lb = pool[-1][0] if len(pool) == ef else float("inf")
        nd = nxt[0] if nxt else float("inf")
        if tie_a is not None and nd > tie_a:
            if lb <= tie_a:
                return None, None, True
            tie_a = None
        if tie_b is not None and lb < tie_b:
            tie_b = None
        if tie_b is not None and nd >= tie_b:
            return None, None, True
        if nxt is None:
            break
        if nxt not in pool:
            # dropped by this expansion's own merge: it lies beyond lowerBound
            # or ties with it, which the checks above have settled
            break
        node = nxt[1]
        done.add(node)
        expanded += 1
    if len(pool) > k and pool[k - 1][0] == pool[k][0]:
        return None, None, True
    return pool[:k], expanded, False


@pytest.mark.parametrize("values", [3, 8, 25, 100, 1000])
def test_unflagged_runs_are_the_references(values):
    rng = random.Random(values)
    kept = 0
    for _ in range(1500):
        n = rng.choice([12, 40, 120])
        degree = rng.choice([3, 6, 10])
        links = [rng.sample(range(n), min(n, degree)) for _ in range(n)]
        # distances that fall along some links, as in a search graph
        dist = [rng.randrange(values) for _ in range(n)]
        ef = rng.choice([1, 2, 5, 10, 25])
        k = rng.randint(1, ef)
        ep = rng.randrange(n)
        got, expanded, matters = id_order(links, dist, ep, ef, k)
        if matters:
            continue
        kept += 1
        want, steps = reference(links, dist, ep, ef, k)
        assert got == want and expanded == steps
    assert kept >= 75
