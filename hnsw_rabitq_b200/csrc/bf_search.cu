// Exact brute-force k-NN on B200 (sm_100a), FP32 in the reference's order.
//
// Replaces BruteforceSearch::searchKnn (hnswlib/bruteforce.h:106-125).  Its
// result is, for every query, the k smallest (distance, label) pairs over the
// allowed rows: the reference's max-heap of std::pair<float, labeltype>
// accepts `dist <= lastdist || size < k` and pops the largest pair, so ties at
// the k-th distance are resolved by label.  These kernels compute the same set
// with the same FP32 distances (the summation orders of device_common.cuh),
// hence bit-identical outputs.
//
// Two launches per batch of queries:
// 1. bf_dist_kernel: a CTA of 128 threads owns 128 rows x QT queries.  Row and
//    query slices of 32 floats stream through a 3-stage cp.async ring, so the
//    shared memory does not depend on the dimension, and a thread keeps all of
//    the reference's accumulators of its row against the QT queries in
//    registers (a row word read from shared memory is used QT times, the query
//    reads are broadcasts).  It writes the distance keys and, per 32 rows, the
//    smallest allowed key.
// 2. bf_select_kernel, one CTA per query: the k-th smallest of 512 group
//    minima bounds the k-th smallest key from above (k rows lie at or below
//    it), so only the few 32-row groups at or below that bound are read, and
//    about 1.1 k keys are sorted by (distance, label).
//
// Query tiles vary fastest over the grid: the CTAs running at one time share
// their rows through L2, so each row comes from HBM once.
//
// Measured (a call from and to host memory): 1 query x 100k rows x 100 dims
// 0.097 ms (scan 12 us, selection 13 us), 1000 x 10k x 128 0.39 ms.  One CTA
// per 32 queries streaming the whole database, with the results kept in its
// shared memory (which left 8-row tiles at 768 dims), took 103 ms and 2.2 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bf_search.h"
#include "device_common.cuh"
#include "launch_cache.h"

namespace hnswgpu {

namespace {

constexpr int kRows = 128;            // rows (= threads) per CTA
constexpr int kKC = 32;               // floats of a row per stage
constexpr int kXStride = kKC + 4;     // 16-byte reads of 8 consecutive rows hit 32 distinct banks
constexpr int kStages = 3;
constexpr int kSelThreads = 512;      // group minima sorted by the selection
constexpr int kSelGroups = 2048;      // 32-row groups the bound may select

// How the reference sums a distance of this dimension (device_common.cuh):
// kAcc16: 16 accumulators over the 16-element blocks, then a scalar tail;
// kAcc4: 4 accumulators (inner product: 8, folded to 4) over 4-element chunks.
enum { kAcc16 = 0, kAcc4 = 1 };

__host__ __device__ inline int dist_form(uint32_t dim) {
    return ((dim & 15) == 0 || (dim > 16 && (dim & 3) != 0)) ? kAcc16 : kAcc4;
}

template <int SPACE, int FORM>
struct Acc {
    static constexpr int N = FORM == kAcc16 ? 16 : (SPACE == 0 ? 4 : 8);
    float a[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N; i++) a[i] = 0.f;
    }
    __device__ __forceinline__ void step(int i, float q, float x) {
        if (SPACE == 0) {
            const float t = __fsub_rn(q, x);
            a[i] = __fmaf_rn(t, t, a[i]);
        } else {
            a[i] = __fmaf_rn(q, x, a[i]);
        }
    }
    // one float4 (chunk u of 4) of a 16-element block
    __device__ __forceinline__ void chunk(int u, const float4& q, const float4& x) {
        step((4 * u + 0) % N, q.x, x.x);
        step((4 * u + 1) % N, q.y, x.y);
        step((4 * u + 2) % N, q.z, x.z);
        step((4 * u + 3) % N, q.w, x.w);
    }
    // the last dim % 16 elements (q, x at their start) and the reduction
    __device__ __forceinline__ float finish(const float* q, const float* x, int dim) {
        const int rem = dim & 15;
        float r;
        if (FORM == kAcc16) {
            if (SPACE == 0) {
                r = a[0];
#pragma unroll
                for (int l = 1; l < N; l++) r = __fadd_rn(r, a[l]);
            } else {
                float t3[8], t6[4];
#pragma unroll
                for (int i = 0; i < 8; i++) t3[i] = __fadd_rn(a[(i + 8) % N], a[i % N]);
#pragma unroll
                for (int i = 0; i < 4; i++) t6[i] = __fadd_rn(t3[i + 4], t3[i]);
                r = __fadd_rn(__fadd_rn(t6[0], t6[2]), __fadd_rn(t6[1], t6[3]));
            }
            if (rem) r = __fadd_rn(r, SPACE == 0 ? l2_scalar(q, x, rem) : ip_scalar(q, x, rem));
        } else {
            if (dim < 4) {
                r = SPACE == 0 ? l2_scalar(q, x, dim) : ip_scalar(q, x, dim);
            } else {
                float s[4];
#pragma unroll
                for (int i = 0; i < 4; i++) s[i] = SPACE == 0 ? a[i] : __fadd_rn(a[i], a[(i + 4) % N]);
                const float4* q4 = reinterpret_cast<const float4*>(q);
                const float4* x4 = reinterpret_cast<const float4*>(x);
                for (int c = 0; c < rem >> 2; c++) {
                    const float4 u = q4[c], v = x4[c];
                    const float uq[4] = {u.x, u.y, u.z, u.w}, vx[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float t = SPACE == 0 ? __fsub_rn(uq[i], vx[i]) : uq[i];
                        s[i] = __fmaf_rn(t, SPACE == 0 ? t : vx[i], s[i]);
                    }
                }
                r = __fadd_rn(__fadd_rn(__fadd_rn(s[0], s[1]), s[2]), s[3]);
                const int r4 = rem & ~3;
                if (rem & 3)
                    r = __fadd_rn(r, SPACE == 0 ? l2_scalar(q + r4, x + r4, rem - r4) : ip_scalar(q + r4, x + r4, rem - r4));
            }
        }
        return SPACE == 0 ? r : __fsub_rn(1.0f, r);
    }
};

__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int bytes, bool valid) {
    const int n = valid ? bytes : 0;  // the rest of the destination is zero filled
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

template <int QT>
struct DistSmem {
    float x[kStages][kRows * kXStride];
    float q[kStages][QT * kKC];
};

// Distance keys of 128 rows x QT queries.  QT = 1 is bound by the loads in
// flight (400k x 100: 34 us, 4.85 TB/s, 74 % of a copy's rate; 15 warps an SM by
// shared memory, 3.5 cycles an issue on global loads).  QT = 8 fills no unit: 100
// queries x 100k x 128 take 226 us with 59 % of the issue slots and 47 % of the
// shared-memory pipe (per 16 elements 16 wavefronts for the row and 4 QT for the
// queries, beside 16 QT FMA and, for L2, 16 QT subtractions); 205 registers and 58
// KB leave 8 warps an SM to hide their latencies.
template <int SPACE, int FORM, int QT>
__global__ void __launch_bounds__(kRows) bf_dist_kernel(BfParams p) {
    extern __shared__ __align__(16) unsigned char raw[];
    DistSmem<QT>& s = *reinterpret_cast<DistSmem<QT>*>(raw);
    const int t = threadIdx.x;
    const uint32_t q_tiles = (p.nq + QT - 1) / QT;
    const uint32_t qb = (uint32_t)(blockIdx.x % q_tiles) * QT;
    const uint64_t r0 = (uint64_t)(blockIdx.x / q_tiles) * kRows;
    const int dim = (int)p.dim;
    const int chunks = ((int)p.row_floats + kKC - 1) / kKC;

    auto load = [&](int c) {
        if (c < chunks) {
            const int stage = c % kStages;
            const int col = c * kKC + (t & 7) * 4;
            const bool in = col < (int)p.row_floats;
#pragma unroll
            for (int i = 0; i < kRows / 16; i++) {
                const int r = (t >> 3) + 16 * i;
                const uint64_t row = min(r0 + r, (uint64_t)p.count - 1);  // rows past the end repeat the last one
                cp_async(smem_u32(&s.x[stage][r * kXStride + (t & 7) * 4]), p.vecs + row * p.row_floats + (in ? col : 0), 16, in);
            }
            for (int i = t; i < QT * kKC; i += kRows) {
                const int e = c * kKC + i % kKC;
                const uint32_t q = min(qb + i / kKC, p.nq - 1);
                const bool ok = e < dim;
                cp_async(smem_u32(&s.q[stage][i]), p.queries + (size_t)q * dim + (ok ? e : 0), 4, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int c = 0; c < kStages - 1; c++) load(c);

    Acc<SPACE, FORM> acc[QT];
#pragma unroll
    for (int j = 0; j < QT; j++) acc[j].zero();
    float d[QT];
    const int n16 = dim >> 4;
    for (int c = 0; c < chunks; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // slice c has landed; every thread is done with slice c - 1
        load(c + kStages - 1);
        const float* x = &s.x[c % kStages][t * kXStride];
        const float* q = &s.q[c % kStages][0];
#pragma unroll
        for (int b = 0; b < kKC / 16; b++) {
            const int blk = c * (kKC / 16) + b;
            if (blk < n16) {
                float4 xv[4];
#pragma unroll
                for (int u = 0; u < 4; u++) xv[u] = reinterpret_cast<const float4*>(x + 16 * b)[u];
#pragma unroll
                for (int j = 0; j < QT; j++)
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        acc[j].chunk(u, reinterpret_cast<const float4*>(q + j * kKC + 16 * b)[u], xv[u]);
            }
            // the tail's block, or past the last full one in the last slice
            if (c == chunks - 1 && (blk == n16 || (blk == n16 - 1 && (dim & 15) == 0))) {
                const int off = blk == n16 ? 16 * b : 0;
#pragma unroll
                for (int j = 0; j < QT; j++) d[j] = acc[j].finish(q + j * kKC + off, x + off, dim);
            }
        }
    }
    const uint64_t row = r0 + t;
    const bool valid = row < p.count;
    const bool allowed = valid && (!p.allow || p.allow[row]);
#pragma unroll
    for (int j = 0; j < QT; j++) {
        const uint32_t q = qb + j;
        if (q >= p.nq) break;
        const uint32_t key = fkey(d[j]);
        if (valid) p.keys[(size_t)q * p.count + row] = key;
        const uint32_t m = __reduce_min_sync(FULL, allowed ? key : 0xffffffffu);
        if ((t & 31) == 0 && valid) p.gmin[(size_t)q * p.groups + (row >> 5)] = m;
    }
}

// Ascending bitonic sort of n (a power of two) (key, label) pairs by a CTA.
__device__ __forceinline__ void sort_pairs(uint32_t* sk, uint64_t* sl, uint32_t n) {
    for (uint32_t size = 2; size <= n; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t h = threadIdx.x; h < n / 2; h += blockDim.x) {
                const uint32_t i = 2 * h - (h & (stride - 1)), j = i + stride;
                const uint32_t ki = sk[i], kj = sk[j];
                const uint64_t li = sl[i], lj = sl[j];
                const bool gt = ki > kj || (ki == kj && li > lj);
                if (gt == ((i & size) == 0)) {
                    sk[i] = kj;
                    sk[j] = ki;
                    sl[i] = lj;
                    sl[j] = li;
                }
            }
            __syncthreads();
        }
}

struct SelShared {
    uint32_t mins[kSelThreads];
    uint32_t list[kSelGroups];
    uint32_t hist[256];
    uint32_t n_list, n_cand, digit, below;
};

// The k best rows of one query by (distance key, label).
__global__ void __launch_bounds__(kSelThreads) bf_select_kernel(BfParams p, uint32_t cap) {
    extern __shared__ __align__(16) unsigned char raw[];
    uint64_t* cl = reinterpret_cast<uint64_t*>(raw);           // cap labels
    uint32_t* ck = reinterpret_cast<uint32_t*>(cl + cap);      // cap keys
    __shared__ SelShared s;
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t q = blockIdx.x;
    const uint32_t* keys = p.keys + (size_t)q * p.count;
    const uint32_t* gmin = p.gmin + (size_t)q * p.groups;
    // ---- the bound: k-th smallest minimum of 512 sets of groups
    uint32_t bound = 0xffffffffu;
    if (p.k <= kSelThreads) {
        uint32_t m = 0xffffffffu;
#pragma unroll 8
        for (uint32_t g = t; g < p.groups; g += kSelThreads) m = min(m, gmin[g]);
        s.mins[t] = m;
        __syncthreads();
        for (uint32_t size = 2; size <= kSelThreads; size <<= 1)
            for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
                const uint32_t j = t ^ stride;
                const uint32_t a = s.mins[t], b = s.mins[j];
                __syncthreads();
                const bool lower = t < (int)j, up = (t & size) == 0;
                s.mins[t] = (lower == up) ? min(a, b) : max(a, b);
                __syncthreads();
            }
        bound = s.mins[p.k - 1];
    }
    if (t == 0) s.n_list = s.n_cand = 0;
    __syncthreads();
    auto put = [&](uint32_t key, uint64_t row) {
        const uint32_t i = atomicAdd(&s.n_cand, 1u);
        if (i < cap) {
            ck[i] = key;
            cl[i] = p.labels[row];
        }
    };
    bool done = false;
    if (bound != 0xffffffffu) {
        for (uint32_t g = t; g < p.groups; g += kSelThreads)
            if (gmin[g] <= bound) {
                const uint32_t i = atomicAdd(&s.n_list, 1u);
                if (i < kSelGroups) s.list[i] = g;
            }
        __syncthreads();
        if (s.n_list <= kSelGroups) {
            for (uint32_t i = t >> 5; i < s.n_list; i += kSelThreads / 32) {
                const uint64_t row = (uint64_t)s.list[i] * 32 + lane;
                if (row < p.count && keys[row] <= bound && (!p.allow || p.allow[row])) put(keys[row], row);
            }
            __syncthreads();
            done = s.n_cand <= cap;
        }
    }
    if (!done) {
        // General form (few rows per result, or more ties than fit): radix
        // selection over all allowed rows, on the key and, among the rows
        // that tie with the k-th key, on the label.
        uint32_t prefix = 0, need = p.k;  // rank still to be found within the prefix
        uint64_t lprefix = 0;
        bool by_label = false, all = false;
        for (int pass = 0; pass < 12 && !all; pass++) {
            const int shift = pass < 4 ? 24 - 8 * pass : 56 - 8 * (pass - 4);
            if (pass == 4) {
                // ties of the k-th key: take them all when they fit
                __syncthreads();
                if (p.k - need + s.below <= cap) break;
                by_label = true;
            }
            __syncthreads();
            for (int i = t; i < 256; i += kSelThreads) s.hist[i] = 0;
            __syncthreads();
            for (uint64_t row = t; row < p.count; row += kSelThreads) {
                if (p.allow && !p.allow[row]) continue;
                const uint32_t key = keys[row];
                if (pass < 4) {
                    if (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8)))
                        atomicAdd(&s.hist[(key >> shift) & 255u], 1u);
                } else if (key == prefix) {
                    const uint64_t lab = p.labels[row];
                    if (pass == 4 || (lab >> (shift + 8)) == (lprefix >> (shift + 8)))
                        atomicAdd(&s.hist[(uint32_t)(lab >> shift) & 255u], 1u);
                }
            }
            __syncthreads();
            if (t == 0) {
                uint32_t sum = 0, digit = 256;
                for (uint32_t i = 0; i < 256; i++) {
                    if (sum + s.hist[i] >= need) {
                        digit = i;
                        break;
                    }
                    sum += s.hist[i];
                }
                s.digit = digit;
                s.n_list = need - sum;                       // rank within the digit
                s.below = digit < 256 ? s.hist[digit] : 0u;  // rows with this prefix
            }
            __syncthreads();
            if (s.digit == 256) {
                all = true;  // fewer than k allowed rows (first pass only)
            } else {
                need = s.n_list;
                if (pass < 4) prefix |= s.digit << shift;
                else lprefix |= (uint64_t)s.digit << shift;
            }
        }
        __syncthreads();
        if (t == 0) s.n_cand = 0;
        __syncthreads();
        for (uint64_t row = t; row < p.count; row += kSelThreads) {
            if (p.allow && !p.allow[row]) continue;
            const uint32_t key = keys[row];
            if (all || key < prefix || (key == prefix && (!by_label || p.labels[row] <= lprefix))) put(key, row);
        }
        __syncthreads();
    }
    const uint32_t n = min(s.n_cand, cap);
    uint32_t P = 1;
    while (P < n) P <<= 1;
    for (uint32_t i = n + t; i < P; i += kSelThreads) {
        ck[i] = 0xffffffffu;
        cl[i] = ~0ull;
    }
    __syncthreads();
    sort_pairs(ck, cl, P);
    const uint32_t kk = min(p.k, n);
    for (uint32_t i = t; i < p.k; i += kSelThreads) {
        p.out_labels[(size_t)q * p.k + i] = i < kk ? cl[i] : ~0ull;
        p.out_dists[(size_t)q * p.k + i] = i < kk ? funkey(ck[i]) : __int_as_float(0x7f800000);
    }
    if (t == 0) p.out_counts[q] = (int32_t)kk;
}

// normalize_vector of every query (cosine), one warp each.
__global__ void bf_normalize_kernel(const float* __restrict__ q, uint32_t nq, int dim, float* __restrict__ out) {
    const uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (r >= nq) return;
    const float* x = q + (size_t)r * dim;
    const float sc = norm_scale(x, dim);
    for (int i = threadIdx.x & 31; i < dim; i += 32) out[(size_t)r * dim + i] = __fmul_rn(x[i], sc);
}

// Capacity of the selection's sort: the k results and their ties.
uint32_t select_cap(uint32_t k) {
    uint32_t c = 1024;
    while (c < 2 * k) c <<= 1;
    return c;
}

template <int SPACE, int FORM, int QT>
cudaError_t launch_dist(const BfParams& p, cudaStream_t stream) {
    static LaunchCache cache;
    const void* fn = (const void*)bf_dist_kernel<SPACE, FORM, QT>;
    int occ = 0;
    cudaError_t e = cache.blocks_per_sm(fn, kRows, sizeof(DistSmem<QT>), &occ);
    if (e != cudaSuccess) return e;
    const uint64_t blocks = (uint64_t)((p.nq + QT - 1) / QT) * ((p.count + kRows - 1) / kRows);
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
    bf_dist_kernel<SPACE, FORM, QT><<<(unsigned)blocks, kRows, sizeof(DistSmem<QT>), stream>>>(p);
    return cudaGetLastError();
}

template <int SPACE, int FORM>
cudaError_t launch_dist_q(const BfParams& p, cudaStream_t stream) {
    // one query keeps 16 accumulators, so more CTAs (bytes in flight) fit an
    // SM; 8 queries per thread halve the row reads per FMA of 4
    if (p.nq == 1) return launch_dist<SPACE, FORM, 1>(p, stream);
    if (p.nq <= 4) return launch_dist<SPACE, FORM, 4>(p, stream);
    return launch_dist<SPACE, FORM, 8>(p, stream);
}

}  // namespace

bool bf_supported(uint32_t k, uint32_t row_floats, size_t max_smem) {
    // The interface's limit on k and the dimension: a fixed function of both
    // (4 queries with their results and sort area beside 16 rows), kept
    // although these kernels' own shared memory grows with neither.
    uint64_t s = 1;
    while (s < (uint64_t)k + 64) s <<= 1;
    uint64_t bytes = (16 + 16ull * row_floats + 127) / 128 * 128;
    bytes = (bytes + 64ull * (row_floats + 4) + 48ull * k + 2048 + 15) / 16 * 16 + 16 + 12 * s;
    return (bytes + 127) / 128 * 128 <= max_smem;
}

static uint64_t bytes_per_query(const BfParams& p) {
    return (uint64_t)p.count * 4 + (uint64_t)((p.count + 31) / 32) * 4;
}

uint32_t bf_batch(const BfParams& p) {
    // 64 MB of distance keys at most (they stay in L2 between the two kernels,
    // and a first call does not wait long for the memory), but no fewer than
    // one tile of queries
    const uint64_t fit = std::max<uint64_t>(8, (64ull << 20) / bytes_per_query(p) / 8 * 8);
    return (uint32_t)std::min<uint64_t>(p.nq, fit);
}

size_t bf_workspace(const BfParams& p, uint32_t batch) {
    return (size_t)batch * bytes_per_query(p) + (p.normalize ? (size_t)p.nq * p.dim * 4 : 0);
}

cudaError_t launch_bf_search(BfParams p, int space, void* workspace, uint32_t batch, cudaStream_t stream) {
    if (p.nq == 0) return cudaSuccess;
    p.groups = (p.count + 31) / 32;
    p.keys = static_cast<uint32_t*>(workspace);
    p.gmin = p.keys + (size_t)batch * p.count;
    cudaError_t e;
    if (p.normalize) {
        float* qn = reinterpret_cast<float*>(p.gmin + (size_t)batch * p.groups);
        bf_normalize_kernel<<<(p.nq + 3) / 4, 128, 0, stream>>>(p.queries, p.nq, (int)p.dim, qn);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        p.queries = qn;
    }
    const uint32_t cap = select_cap(p.k);
    static LaunchCache cache;
    int occ = 0;
    e = cache.blocks_per_sm((const void*)bf_select_kernel, kSelThreads, (size_t)cap * 12, &occ);
    if (e != cudaSuccess) return e;
    for (uint32_t b = 0; b < p.nq; b += batch) {
        BfParams c = p;
        c.nq = std::min(batch, p.nq - b);
        c.queries = p.queries + (size_t)b * p.dim;
        c.out_labels = p.out_labels + (size_t)b * p.k;
        c.out_dists = p.out_dists + (size_t)b * p.k;
        c.out_counts = p.out_counts + b;
        if (dist_form(p.dim) == kAcc16)
            e = space == 0 ? launch_dist_q<0, kAcc16>(c, stream) : launch_dist_q<1, kAcc16>(c, stream);
        else
            e = space == 0 ? launch_dist_q<0, kAcc4>(c, stream) : launch_dist_q<1, kAcc4>(c, stream);
        if (e != cudaSuccess) return e;
        bf_select_kernel<<<c.nq, kSelThreads, (size_t)cap * 12, stream>>>(c, cap);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace hnswgpu
