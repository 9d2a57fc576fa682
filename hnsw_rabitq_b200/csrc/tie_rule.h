// When a run in the (distance, id) order has the result of the reference's
// run, whose two heaps order equal distances by their layout
// (hnswlib/hnswalg.h:321-322).  The tie-exact beam runs without heaps and
// repeats a query with them only when this rule says that a tie can matter.
// Usable from host code for testing.
//
// Acceptance is by counting and does not depend on heap layout, so the two
// runs differ only where distances tie:
//   (a) The candidate popped next shares its distance d with another one.  Both
//       runs then expand the tied candidates and everything they find at d or
//       closer, in different orders, before they go beyond d.  If lowerBound is
//       still above d when that is done, every one of these nodes was accepted
//       and expanded in either order (lowerBound only falls), so the same nodes
//       have been seen.  When, besides, no node at exactly lowerBound has been
//       left out of the full pool meanwhile, the pool holds every node at
//       lowerBound or closer that it held before or that was seen meanwhile:
//       exactly ef, hence the same ef in any order, none of which either run can
//       have rejected.  What the runs accepted differently lies beyond
//       lowerBound, where a candidate can only end the search.  A node left out
//       at lowerBound was either dropped from the pool (that is (b)) or rejected,
//       and then at a lowerBound that did not fall any further: it equals the
//       bound AFTER the unit of neighbours that rejected it.  (The bound before
//       the unit is not enough: neighbours of the same unit lower it for those
//       behind them.)
//   (b) The entry dropped from the full pool ties with its new worst entry.
//       The reference may keep the other one, and both stay in its
//       candidate_set; that matters only if candidates at that distance come up
//       for expansion (or the search ends) while lowerBound is still there.
//   (c) The k-th and the next result tie: the heap's layout decides (the
//       caller's check, on the final pool).
#pragma once
#include <cstdint>

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#ifndef __forceinline__
#define __forceinline__ inline
#endif
#endif

namespace hnswgpu {

// Distances are the order-preserving unsigned keys of the beam; kNoBound
// stands for "the pool is not full" and "no candidate left".
struct TieRule {
    static constexpr uint32_t kNoBound = 0xffffffffu;
    uint32_t a = 0, b = 0;  // distances of the ties (a), (b) not settled yet (0: none)
    bool matters = false;

    // Whether neighbours rejected by the unit about to be taken can matter.
    __host__ __device__ __forceinline__ bool open() const { return a != 0; }
    // A unit taken while open() rejected a neighbour at exactly the bound after it.
    __host__ __device__ __forceinline__ void rejected() { matters = true; }
    // The next candidate, at distance nd, is one of `same` at that distance.
    __host__ __device__ __forceinline__ void picked(uint32_t nd, int same) {
        if (same > 1 && nd > a) a = nd;
    }
    // A unit's merge dropped entries, the closest at `dropped`; lb: the bound now.
    __host__ __device__ __forceinline__ void dropped(uint32_t closest, uint32_t lb) {
        if (closest == lb) b = closest;
    }
    // After an expansion: lb the bound now, nd the next candidate's distance.
    __host__ __device__ __forceinline__ void settle(uint32_t lb, uint32_t nd) {
        if (a && nd > a) {
            if (lb <= a) matters = true;
            a = 0;
        }
        if (lb < b) b = 0;
        if (b && nd >= b) matters = true;
    }
};

}  // namespace hnswgpu
