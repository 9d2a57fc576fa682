// The rule of hnsw_rabitq_b200/csrc/tie_rule.h against the reference's two
// heaps (ref_heap.h), on small graphs whose distances tie: a run in the
// (distance, id) order that meets no tie that can matter must have the
// reference's results and expansions.  The id-order run is the beam's: a list
// is taken in units of neighbours (32 in the kernel, fewer here), each with the
// reference's sequential acceptance test.  Fixed cases first, then random
// graphs until argv[1] runs were kept.  Prints "ok <runs> <kept>" or the first
// difference.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "ref_heap.h"
#include "tie_rule.h"

using hnswgpu::CandLess;
using hnswgpu::TieRule;
using hnswgpu::TopLess;
typedef std::vector<std::vector<uint32_t>> Links;

struct Run {
    std::vector<uint64_t> result;  // (distance << 32 | id), ascending
    int expanded = 0;
    bool matters = false;
};

static uint32_t hi(uint64_t e) { return (uint32_t)(e >> 32); }
static uint64_t entry(const std::vector<uint32_t>& dist, uint32_t id) { return ((uint64_t)dist[id] << 32) | id; }

static Run reference(const Links& links, const std::vector<uint32_t>& dist, uint32_t ep, int ef, int k) {
    std::vector<uint64_t> top(dist.size() + 2), cand(dist.size() + 2);
    std::vector<char> seen(dist.size(), 0);
    int tn = 0, cn = 0;
    hnswgpu::ref_heap_push(top.data(), tn, entry(dist, ep), TopLess());
    hnswgpu::ref_heap_push(cand.data(), cn, entry(dist, ep), CandLess());
    seen[ep] = 1;
    Run r;
    while (cn > 0 && hi(cand[0]) <= hi(top[0])) {
        const uint32_t c = (uint32_t)hnswgpu::ref_heap_pop(cand.data(), cn, CandLess());
        r.expanded++;
        for (uint32_t x : links[c]) {
            if (seen[x]) continue;
            seen[x] = 1;
            if (tn < ef || hi(top[0]) > dist[x]) {
                hnswgpu::ref_heap_push(cand.data(), cn, entry(dist, x), CandLess());
                hnswgpu::ref_heap_push(top.data(), tn, entry(dist, x), TopLess());
                if (tn > ef) hnswgpu::ref_heap_pop(top.data(), tn, TopLess());
            }
        }
    }
    while (tn > k) hnswgpu::ref_heap_pop(top.data(), tn, TopLess());
    r.result.assign(top.begin(), top.begin() + tn);
    std::sort(r.result.begin(), r.result.end());
    return r;
}

static Run id_order(const Links& links, const std::vector<uint32_t>& dist, uint32_t ep, int ef, int k, int unit) {
    std::vector<uint64_t> pool{entry(dist, ep)};
    std::vector<char> seen(dist.size(), 0), done(dist.size(), 0);
    seen[ep] = done[ep] = 1;
    Run r;
    r.expanded = 1;
    TieRule tie;
    uint32_t node = ep;
    size_t at = 0;
    while (true) {
        const std::vector<uint32_t>& l = links[node];
        const size_t end = std::min(l.size(), at + unit);
        const bool full = (int)pool.size() == ef, open = tie.open();
        const uint32_t lbk = full ? hi(pool.back()) : TieRule::kNoBound;
        std::vector<uint32_t> fresh, rejected;
        std::vector<uint64_t> accepted, live;
        for (; at < end; at++)
            if (!seen[l[at]]) {
                seen[l[at]] = 1;
                fresh.push_back(l[at]);
            }
        for (uint32_t x : fresh) {
            bool ok = !(full && dist[x] >= lbk);
            if (ok) {
                int closer = 0;
                for (uint64_t e : pool) closer += hi(e) <= dist[x];
                for (uint64_t e : live) closer += hi(e) <= dist[x];
                live.push_back(entry(dist, x));
                ok = closer < ef;
            }
            if (ok) accepted.push_back(entry(dist, x));
            else rejected.push_back(x);
        }
        const bool inner = at < l.size();
        // the next candidate: the closest unexpanded one, by (distance, id)
        uint64_t next = ~0ull;
        if (!inner) {
            for (uint64_t e : pool)
                if (!done[(uint32_t)e]) next = std::min(next, e);
            for (uint64_t e : accepted) next = std::min(next, e);
            if (next != ~0ull) {
                int same = 0;
                for (uint64_t e : pool) same += !done[(uint32_t)e] && hi(e) == hi(next);
                for (uint64_t e : accepted) same += hi(e) == hi(next);
                tie.picked(hi(next), same);
            }
        }
        pool.insert(pool.end(), accepted.begin(), accepted.end());
        std::sort(pool.begin(), pool.end());
        if ((int)pool.size() > ef) {
            tie.dropped(hi(pool[ef]), hi(pool[ef - 1]));
            pool.resize(ef);
        }
        const uint32_t lb = (int)pool.size() == ef ? hi(pool.back()) : TieRule::kNoBound;
        if (open)
            for (uint32_t x : rejected)
                if (dist[x] == lb) tie.rejected();
        if (!inner) tie.settle(lb, next == ~0ull ? TieRule::kNoBound : hi(next));
        if (tie.matters) {
            r.matters = true;
            return r;
        }
        if (inner) continue;
        if (next == ~0ull) break;
        node = (uint32_t)next;
        at = 0;
        done[node] = 1;
        r.expanded++;
    }
    if ((int)pool.size() > k && hi(pool[k - 1]) == hi(pool[k])) {
        r.matters = true;
        return r;
    }
    r.result.assign(pool.begin(), pool.begin() + std::min<size_t>(k, pool.size()));
    return r;
}

static long runs = 0, kept = 0;

static bool check(const Links& links, const std::vector<uint32_t>& dist, uint32_t ep, int ef, int k, int unit) {
    const Run mine = id_order(links, dist, ep, ef, k, unit);
    runs++;
    if (mine.matters) return true;
    kept++;
    const Run want = reference(links, dist, ep, ef, k);
    if (mine.result == want.result && mine.expanded == want.expanded) return true;
    std::printf("difference: ef %d k %d unit %d entry %u, %d and %d expansions\n", ef, k, unit, ep, mine.expanded,
                want.expanded);
    for (size_t i = 0; i < links.size(); i++) {
        std::printf("  %zu (distance %u):", i, dist[i]);
        for (uint32_t x : links[i]) std::printf(" %u", x);
        std::printf("\n");
    }
    return false;
}

// A neighbour rejected at the bound that an earlier one of its own unit has
// lowered, while two candidates tie: two graphs, with every order of a list.
static bool fixed() {
    const Links a = {{5, 1, 7, 6, 4}, {4, 6, 5, 7, 0}, {6, 3, 4, 0, 5}, {4, 7, 6, 2, 0},
                     {0, 2, 3, 6, 7}, {4, 7, 1, 6, 0}, {3, 4, 1, 2, 0}, {6, 4, 5, 1, 0}};
    const std::vector<uint32_t> da = {2, 3, 2, 2, 1, 3, 1, 3};  // (a distance key is not 0)
    const Links b = {{2, 1, 3, 4}, {5}, {6, 7}, {}, {}, {}, {}, {}};
    const std::vector<uint32_t> db = {50, 10, 10, 40, 45, 30, 20, 30};
    for (int which = 0; which < 2; which++) {
        Links l = which ? b : a;
        for (auto& order : {0, 1, 2, 3, 4, 5, 6, 7}) {
            std::vector<uint32_t> sorted = l[order];
            std::sort(sorted.begin(), sorted.end());
            do {
                Links m = l;
                m[order] = sorted;
                for (int ef = 1; ef <= 8; ef++)
                    for (int k = 1; k <= ef; k++)
                        for (int unit : {2, 3, 32})
                            if (!check(m, which ? db : da, 0, ef, k, unit)) return false;
            } while (std::next_permutation(sorted.begin(), sorted.end()));
        }
    }
    return true;
}

int main(int argc, char** argv) {
    const long want = argc > 1 ? std::atol(argv[1]) : 100000;
    if (!fixed()) return 1;
    kept = 0;
    std::mt19937 rng(12345);
    auto below = [&](uint32_t n) { return (uint32_t)(rng() % n); };
    while (kept < want) {
        const uint32_t n = 6 + below(below(4) ? 20 : 90);
        const uint32_t degree = 2 + below(9);
        const uint32_t values = 2 + below(below(2) ? 10 : 60);
        const int kind = (int)below(3);
        std::vector<uint32_t> dist(n);
        Links links(n);
        if (kind == 2) {
            // rows of small integers: nearest-neighbour links and a few random ones
            const uint32_t dim = 1 + below(6);
            std::vector<uint32_t> x(n * dim), q(dim);
            for (auto& v : x) v = below(values);
            for (auto& v : q) v = below(values);
            auto d2 = [&](const uint32_t* u, const uint32_t* v) {
                uint32_t s = 0;
                for (uint32_t i = 0; i < dim; i++) s += (u[i] - v[i]) * (u[i] - v[i]);
                return s;
            };
            for (uint32_t i = 0; i < n; i++) dist[i] = d2(&x[i * dim], q.data()) + 1;
            std::vector<uint32_t> order(n), to(n);
            for (uint32_t i = 0; i < n; i++) {
                for (uint32_t j = 0; j < n; j++) {
                    order[j] = j;
                    to[j] = j == i ? ~0u : d2(&x[i * dim], &x[j * dim]);
                }
                std::stable_sort(order.begin(), order.end(), [&](uint32_t u, uint32_t v) { return to[u] < to[v]; });
                for (uint32_t j = 0; j < std::min(degree, n - 1); j++) links[i].push_back(order[j]);
                const uint32_t extra = below(n);
                if (extra != i && std::find(links[i].begin(), links[i].end(), extra) == links[i].end())
                    links[i].push_back(extra);
                std::shuffle(links[i].begin(), links[i].end(), rng);
            }
        } else {
            for (auto& v : dist) v = 1 + below(values);
            for (uint32_t i = 0; i < n; i++) {
                std::vector<uint32_t> pick;
                for (uint32_t t = 0; t < 4 * degree && pick.size() < degree; t++) {
                    const uint32_t x = below(n);
                    if (x == i || std::find(pick.begin(), pick.end(), x) != pick.end()) continue;
                    // kind 1: distances fall along most links, as in a search graph
                    if (kind == 1 && dist[x] > dist[i] && below(4)) continue;
                    pick.push_back(x);
                }
                links[i] = pick;
            }
        }
        const uint32_t ep = below(n);
        for (int t = 0; t < 4; t++) {
            const int ef = 1 + (int)below(10), k = below(3) ? ef : 1 + (int)below(ef);
            const int units[] = {2, 3, 5, 32};
            if (!check(links, dist, ep, ef, k, units[t])) return 1;
        }
    }
    std::printf("ok %ld %ld\n", runs, kept);
    return 0;
}
