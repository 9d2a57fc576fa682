// Training of the early-termination network on the GPU (sm_100a): forward,
// backward and Adam kernels, plus the stand-alone inference kernel that runs
// the search's own in-warp network on given feature vectors.
//
// Network: x = (f - mu) * inv_sigma; h1 = relu(W1 x + b1); h2 = relu(W2 h1 + b2);
// logit = w3 . h2 + b3.  Loss: class-weighted binary cross-entropy,
//   pos_weight * y * softplus(-logit) + (1 - y) * softplus(logit),
// averaged over the batch.  Parameters are float32 (kTermParams, layout in
// hnsw_search.h); mu / inv_sigma are fixed by the caller and get no gradient.
//
// term_grad_kernel: four CTAs of 512 threads per 128 samples, four threads per
// sample for the forward and the activation gradients (activations kept in
// shared memory, rows padded to 65 floats so the per-sample rows fall in
// distinct banks); then each CTA reduces a quarter of the weight gradients over
// the samples into the tile's partial-gradient row.  term_epoch_kernel runs a
// whole epoch of such steps in one cooperative launch: after each batch's
// gradients it sums the rows in a fixed order (deterministic) and applies Adam.
// The sizes are tiny (4.7k parameters), so CUDA cores, not tensor cores, do this
// work.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <numeric>
#include <random>
#include <vector>

#include "hnsw_search.h"
#include "term_mlp.cuh"

namespace hnswgpu {

void pack_term_model(const float* params, unsigned char* out) {
    float* f = reinterpret_cast<float*>(out);
    for (int i = 0; i < kTermPackedFloats; i++) f[i] = 0.f;
    for (int i = 0; i < kTermFeatures; i++) {
        f[i] = params[kTermOffMu + i];
        f[kTermFeatures + i] = params[kTermOffInvSigma + i];
    }
    f[2 * kTermFeatures] = params[kTermOffB3];
    float* b1f = f + kTermPackedHead;
    float* b2f = b1f + 4 * 8 * 2;
    for (int t = 0; t < 4; t++)
        for (int v = 0; v < 8; v++)
            for (int e = 0; e < 2; e++) {
                b1f[(t * 8 + v) * 2 + e] = params[kTermOffB1 + 8 * v + 2 * t + e];
                b2f[(t * 8 + v) * 2 + e] = params[kTermOffB2 + 8 * v + 2 * t + e];
            }
    __half* h = reinterpret_cast<__half*>(out + (size_t)kTermPackedFloats * 4);
    // w3f[t][v]
    for (int t = 0; t < 4; t++)
        for (int v = 0; v < 8; v++)
            for (int e = 0; e < 2; e++) h[(t * 8 + v) * 2 + e] = __float2half_rn(params[kTermOffW3 + 8 * v + 2 * t + e]);
    h += 4 * 8 * 2;
    // W1f[lane][v][hh]
    for (int lane = 0; lane < 32; lane++) {
        const int g = lane >> 2, t = lane & 3;
        for (int v = 0; v < 8; v++)
            for (int hh = 0; hh < 2; hh++)
                for (int e = 0; e < 2; e++) {
                    const int feat = 2 * t + 8 * hh + e;
                    h[((lane * 8 + v) * 2 + hh) * 2 + e] =
                        __float2half_rn(params[kTermOffW1 + (8 * v + g) * kTermFeatures + feat]);
                }
    }
    h += 32 * 8 * 2 * 2;
    // W2f[lane][s][v][hh]
    for (int lane = 0; lane < 32; lane++) {
        const int g = lane >> 2, t = lane & 3;
        for (int st = 0; st < 4; st++)
            for (int v = 0; v < 8; v++)
                for (int hh = 0; hh < 2; hh++)
                    for (int e = 0; e < 2; e++) {
                        const int j = 16 * st + 2 * t + 8 * hh + e;
                        h[(((lane * 4 + st) * 8 + v) * 2 + hh) * 2 + e] =
                            __float2half_rn(params[kTermOffW2 + (8 * v + g) * kTermHidden + j]);
                    }
    }
}

namespace {

constexpr int kTile = 128;             // samples per tile (one partial gradient)
constexpr int kGradThreads = 512;      // 4 threads per sample
constexpr int kSplit = 4;              // CTAs per tile, each writes a quarter of the units' gradients
constexpr int kUnits = kTermHidden / 4;  // units per thread, and per CTA of a tile
constexpr int kRow = kTermHidden + 1;  // padded activation row
constexpr int kXRow = kTermFeatures + 1;
constexpr int kWRow = kTermHidden + 4;  // transposed weights: 16-byte rows, 8 banks to a column
static_assert(kGradThreads == 4 * kTile && kUnits * kSplit == kTermHidden && kUnits == kGradThreads / 32, "gradient tiling");

struct TrainSmem {
    float W1[kTermHidden * kTermFeatures];
    float b1[kTermHidden];
    float W2[kTermHidden * kTermHidden];
    float W2t[kTermHidden * kWRow];  // [input][unit]
    float b2[kTermHidden];
    float w3[kTermHidden];
    float x[kTile * kXRow];
    float dl[kTile];
    float h1[kTile * kRow];
    float h2[kTile * kRow];
    float dz1[kTile * kRow];
    float dz2[kTile * kRow];
    float loss[kTile / 32];
};

// acc[v] = fma(w[v], a, acc[v]) for kUnits consecutive weights (16-byte
// aligned; the same address in every lane).
__device__ __forceinline__ void fma_units(const float* w, float a, float (&acc)[kUnits]) {
#pragma unroll
    for (int v = 0; v < kUnits; v += 4) {
        const float4 q = *reinterpret_cast<const float4*>(w + v);
        acc[v] = fmaf(q.x, a, acc[v]);
        acc[v + 1] = fmaf(q.y, a, acc[v + 1]);
        acc[v + 2] = fmaf(q.z, a, acc[v + 2]);
        acc[v + 3] = fmaf(q.w, a, acc[v + 3]);
    }
}

// Partial gradient of samples [start + 128 * blockIdx.x, ...) of the order
// `perm` (identity when null), scaled by `scale` (1 / batch size).
//
// A batch of 1024 is 8 tiles, so what bounds a step is one CTA's latency: with
// a thread per sample each of the 64 units was a chain of 64 dependent FMAs
// (88 us a step).  Four threads share a sample, each with 16 units side by
// side in registers, and four CTAs share a tile: all compute its activations,
// each writes the gradients of 16 units.  Every sum keeps its order (inputs or
// samples ascending), so the results are the same bits.  27 us a step now, and
// 22.8 -> 9 ms for 4 epochs over 60k samples with the host's part below.
__device__ __forceinline__ void grad_tile(TrainSmem& s, const float* params, const float* __restrict__ feats,
                                          const float* __restrict__ labels, const uint32_t* __restrict__ perm,
                                          uint64_t start, uint64_t end, float pos_weight, float scale, float* part,
                                          float* part_loss, uint32_t tile, uint32_t quarter) {
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    for (int i = t; i < kTermHidden * kTermFeatures; i += kGradThreads) s.W1[i] = __ldcg(params + kTermOffW1 + i);
    for (int i = t; i < kTermHidden * kTermHidden; i += kGradThreads) {
        const float w = __ldcg(params + kTermOffW2 + i);
        s.W2[i] = w;
        s.W2t[(i % kTermHidden) * kWRow + i / kTermHidden] = w;
    }
    if (t < kTermHidden) {
        s.b1[t] = __ldcg(params + kTermOffB1 + t);
        s.b2[t] = __ldcg(params + kTermOffB2 + t);
        s.w3[t] = __ldcg(params + kTermOffW3 + t);
    }
    const float b3 = __ldcg(params + kTermOffB3);
    const uint64_t base = start + (uint64_t)tile * kTile;
    for (int i = t; i < kTile * kTermFeatures; i += kGradThreads) {
        const int r = i / kTermFeatures, f = i % kTermFeatures;
        const bool valid = base + r < end;
        const uint64_t sample = valid ? (perm ? perm[base + r] : base + r) : 0;
        s.x[r * kXRow + f] = valid ? (feats[sample * kTermFeatures + f] - __ldcg(params + kTermOffMu + f)) * __ldcg(params + kTermOffInvSigma + f)
                                   : 0.f;
    }
    __syncthreads();
    // ---- forward: lane's sample r, this warp's units [u0, u0 + 16)
    const int r = (warp & 3) * 32 + lane, u0 = (warp >> 2) * kUnits;
    float* h1 = s.h1 + r * kRow;
    float* h2 = s.h2 + r * kRow;
    float acc[kUnits];
    {
        float x[kTermFeatures];
#pragma unroll
        for (int i = 0; i < kTermFeatures; i++) x[i] = s.x[r * kXRow + i];
#pragma unroll 4
        for (int v = 0; v < kUnits; v++) {
            float a = s.b1[u0 + v];
#pragma unroll
            for (int i = 0; i < kTermFeatures; i++) a = fmaf(s.W1[(u0 + v) * kTermFeatures + i], x[i], a);
            h1[u0 + v] = fmaxf(a, 0.f);
        }
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < kUnits; v++) acc[v] = s.b2[u0 + v];
#pragma unroll 4
    for (int j = 0; j < kTermHidden; j++) fma_units(s.W2t + j * kWRow + u0, h1[j], acc);
#pragma unroll
    for (int v = 0; v < kUnits; v++) h2[u0 + v] = fmaxf(acc[v], 0.f);
    __syncthreads();
    if (t < kTile) {
        // ---- loss and d loss / d logit, one thread per sample
        const bool valid = base + t < end;
        const uint64_t sample = valid ? (perm ? perm[base + t] : base + t) : 0;
        const float* h = s.h2 + t * kRow;
        float logit = b3;
#pragma unroll 16
        for (int u = 0; u < kTermHidden; u++) logit = fmaf(s.w3[u], h[u], logit);
        const float y = valid ? labels[sample] : 0.f;
        const float sp_pos = fmaxf(logit, 0.f) + log1pf(expf(-fabsf(logit)));  // softplus(logit)
        const float sp_neg = sp_pos - logit;                                   // softplus(-logit)
        const float prob = 1.f / (1.f + expf(-logit));
        float loss = valid ? pos_weight * y * sp_neg + (1.f - y) * sp_pos : 0.f;
        const float g = valid ? (pos_weight * y * (prob - 1.f) + (1.f - y) * prob) * scale : 0.f;
        s.dl[t] = g;
#pragma unroll
        for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (lane == 0) s.loss[t >> 5] = loss;
    }
    __syncthreads();
    // ---- backward through the hidden layers
    {
        float* dz2 = s.dz2 + r * kRow;
        const float g = s.dl[r];
#pragma unroll
        for (int v = 0; v < kUnits; v++) dz2[u0 + v] = h2[u0 + v] > 0.f ? g * s.w3[u0 + v] : 0.f;
        __syncthreads();
#pragma unroll
        for (int v = 0; v < kUnits; v++) acc[v] = 0.f;
#pragma unroll 4
        for (int u = 0; u < kTermHidden; u++) fma_units(s.W2 + u * kTermHidden + u0, dz2[u], acc);
        float* dz1 = s.dz1 + r * kRow;
#pragma unroll
        for (int v = 0; v < kUnits; v++) dz1[u0 + v] = h1[u0 + v] > 0.f ? acc[v] : 0.f;
    }
    __syncthreads();
    // ---- weight gradients, summed over the tile's samples: units [q0, q0 + 16)
    float* out = part + (size_t)tile * kTermParams;
    const int q0 = quarter * kUnits;
    {
        // a warp per unit, two inputs per lane
        const int u = q0 + warp;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 8
        for (int i = 0; i < kTile; i++) {
            const float z = s.dz2[i * kRow + u];
            a0 = fmaf(z, s.h1[i * kRow + lane], a0);
            a1 = fmaf(z, s.h1[i * kRow + lane + 32], a1);
        }
        out[kTermOffW2 + u * kTermHidden + lane] = a0;
        out[kTermOffW2 + u * kTermHidden + lane + 32] = a1;
    }
    if (t < kUnits * kTermFeatures) {
        const int u = q0 + t / kTermFeatures, f = t % kTermFeatures;
        float a = 0.f;
#pragma unroll 8
        for (int i = 0; i < kTile; i++) a = fmaf(s.dz1[i * kRow + u], s.x[i * kXRow + f], a);
        out[kTermOffW1 + u * kTermFeatures + f] = a;
    } else if (t < kUnits * kTermFeatures + 32) {
        // biases of the two hidden layers
        const int u = q0 + (lane & (kUnits - 1));
        const float* dz = lane < kUnits ? s.dz1 : s.dz2;
        float a = 0.f;
#pragma unroll 8
        for (int i = 0; i < kTile; i++) a += dz[i * kRow + u];
        out[(lane < kUnits ? kTermOffB1 : kTermOffB2) + u] = a;
    } else if (t < kUnits * kTermFeatures + 64) {
        if (lane < kUnits) {
            const int u = q0 + lane;
            float a = 0.f;
#pragma unroll 8
            for (int i = 0; i < kTile; i++) a = fmaf(s.dl[i], s.h2[i * kRow + u], a);
            out[kTermOffW3 + u] = a;
        }
    } else if (quarter == 0) {
        const int v = t - kUnits * kTermFeatures - 64;
        if (v == 0) {
            float a = 0.f;
#pragma unroll 8
            for (int i = 0; i < kTile; i++) a += s.dl[i];
            out[kTermOffB3] = a;
            float l = 0.f;
            for (int w = 0; w < kTile / 32; w++) l += s.loss[w];
            part_loss[tile] = l * scale;
        } else if (v >= 32 && v < 32 + 2 * kTermFeatures) {
            out[kTermOffMu + (v - 32)] = 0.f;  // mu, inv_sigma: fixed
        }
    }
}

__global__ void __launch_bounds__(kGradThreads) term_grad_kernel(const float* params, const float* feats,
                                                                 const float* labels, uint64_t n, float pos_weight,
                                                                 float scale, float* part, float* part_loss) {
    extern __shared__ __align__(16) unsigned char raw[];
    grad_tile(*reinterpret_cast<TrainSmem*>(raw), params, feats, labels, nullptr, 0, n, pos_weight, scale, part,
              part_loss, blockIdx.x, blockIdx.y);
}

// Sum of the partial rows, in block order (no atomics: deterministic).
__global__ void term_reduce_kernel(const float* __restrict__ part, const float* __restrict__ part_loss, int nparts,
                                   float* __restrict__ grad, float* __restrict__ loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kTermParams) {
        float a = 0.f;
        for (int b = 0; b < nparts; b++) a += part[(size_t)b * kTermParams + i];
        grad[i] = a;
    }
    if (i == 0) {
        float l = 0.f;
        for (int b = 0; b < nparts; b++) l += part_loss[b];
        *loss = l;
    }
}

struct TrainArgs {
    float *params, *m, *v;
    const float *feats, *labels;
    const uint32_t* perm;
    uint64_t n;
    uint32_t batch;
    float lr, pos_weight, wd;
    const float2* bias;    // per batch: Adam's bias corrections
    float *part, *part_loss, *epoch_loss;
    uint32_t *barrier, *failed;
    uint32_t gen;          // barriers passed by earlier launches
};

// Adam over the trainable parameters (W1 onwards), decoupled weight decay
// on the weight matrices; also accumulates the batch loss into `epoch_loss`.
// Thread i of the grid has parameter i.
__device__ __forceinline__ void adam_step(const TrainArgs& a, int i, int nparts, float bc1, float bc2) {
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    if (i == 0) {
        float l = 0.f;
        for (int b = 0; b < nparts; b++) l += __ldcg(a.part_loss + b);
        *a.epoch_loss += l;
    }
    if (i < kTermOffW1 || i >= kTermParams) return;
    float g = 0.f;
    for (int b = 0; b < nparts; b++) g += __ldcg(a.part + (size_t)b * kTermParams + i);
    const float mi = beta1 * a.m[i] + (1.f - beta1) * g;
    const float vi = beta2 * a.v[i] + (1.f - beta2) * g * g;
    a.m[i] = mi;
    a.v[i] = vi;
    const bool is_weight = (i >= kTermOffW1 && i < kTermOffB1) || (i >= kTermOffW2 && i < kTermOffB2) ||
                           (i >= kTermOffW3 && i < kTermOffB3);
    float p = a.params[i];
    if (is_weight) p -= a.lr * a.wd * p;
    p -= a.lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    a.params[i] = p;
}

// All CTAs of a cooperative launch meet; false when the (bounded, seconds)
// wait gave up.
__device__ __forceinline__ bool grid_meet(const TrainArgs& a, uint32_t gen) {
    __shared__ uint32_t ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(a.barrier, 1u);
        const uint32_t want = gen * gridDim.x;
        ok = 0;
        for (uint32_t i = 0; i < (1u << 24); i++)
            if ((int32_t)(*(volatile uint32_t*)a.barrier - want) >= 0) {
                ok = 1;
                break;
            }
        if (!ok) atomicOr(a.failed, 1u);
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// One epoch in one cooperative launch: a step (gradient tiles, then Adam) is
// 20-27 us, and two launches a step cost as much again on a slow host.  Bound by
// one tile's latency: 32 of 148 SMs, 16 warps each, waits for shared memory (3.6
// cycles an issue) and at barriers (2.3).
__global__ void __launch_bounds__(kGradThreads) term_epoch_kernel(TrainArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    TrainSmem& s = *reinterpret_cast<TrainSmem*>(raw);
    uint32_t gen = a.gen;
    uint64_t step = 0;
    for (uint64_t b0 = 0; b0 < a.n; b0 += a.batch, step++) {
        const uint64_t b1 = min(a.n, b0 + a.batch);
        const uint32_t tiles = (uint32_t)((b1 - b0 + kTile - 1) / kTile);
        for (uint32_t w = blockIdx.x; w < tiles * kSplit; w += gridDim.x) {
            grad_tile(s, a.params, a.feats, a.labels, a.perm, b0, b1, a.pos_weight, 1.0f / (float)(b1 - b0), a.part,
                      a.part_loss, w / kSplit, w % kSplit);
            __syncthreads();
        }
        if (!grid_meet(a, ++gen)) return;
        const float2 bias = a.bias[step];
        for (int i = blockIdx.x * kGradThreads + threadIdx.x; i < kTermParams; i += gridDim.x * kGradThreads)
            adam_step(a, i, (int)tiles, bias.x, bias.y);
        if (!grid_meet(a, ++gen)) return;
    }
}

// One warp per feature vector: the search's own inference function.
__global__ void term_logits_kernel(const float* __restrict__ model, const float* __restrict__ feats, uint64_t n,
                                   float* __restrict__ out) {
    const uint64_t row = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    float f[kTermFeatures];
#pragma unroll
    for (int i = 0; i < kTermFeatures; i++) f[i] = feats[row * kTermFeatures + i];
    const float l = term_logit(model, f, lane);
    if (lane == 0) out[row] = l;
}

template <typename T>
struct DevArray {
    T* p = nullptr;
    cudaError_t alloc(size_t n) { return cudaMalloc((void**)&p, std::max<size_t>(n, 1) * sizeof(T)); }
    ~DevArray() {
        if (p) cudaFree(p);
    }
};

#define TERM_CHECK(x)                          \
    do {                                       \
        cudaError_t e_ = (x);                  \
        if (e_ != cudaSuccess) return e_;      \
    } while (0)

}  // namespace

cudaError_t term_loss_grad(const float* params, const float* feats, const float* labels, uint64_t n,
                           float pos_weight, float* out_loss, float* out_grad) {
    DevArray<float> dp, df, dy, dpart, dpl, dg, dl;
    const uint64_t blocks = (n + kTile - 1) / kTile;
    TERM_CHECK(dp.alloc(kTermParams));
    TERM_CHECK(df.alloc(n * kTermFeatures));
    TERM_CHECK(dy.alloc(n));
    TERM_CHECK(dpart.alloc(blocks * kTermParams));
    TERM_CHECK(dpl.alloc(blocks));
    TERM_CHECK(dg.alloc(kTermParams));
    TERM_CHECK(dl.alloc(1));
    TERM_CHECK(cudaMemcpy(dp.p, params, kTermParams * 4, cudaMemcpyHostToDevice));
    TERM_CHECK(cudaMemcpy(df.p, feats, n * kTermFeatures * 4, cudaMemcpyHostToDevice));
    TERM_CHECK(cudaMemcpy(dy.p, labels, n * 4, cudaMemcpyHostToDevice));
    const int smem = (int)sizeof(TrainSmem);
    TERM_CHECK(cudaFuncSetAttribute(term_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    term_grad_kernel<<<dim3((unsigned)blocks, kSplit), kGradThreads, smem>>>(dp.p, df.p, dy.p, n, pos_weight,
                                                                            1.0f / (float)n, dpart.p, dpl.p);
    TERM_CHECK(cudaGetLastError());
    term_reduce_kernel<<<(kTermParams + 255) / 256, 256>>>(dpart.p, dpl.p, (int)blocks, dg.p, dl.p);
    TERM_CHECK(cudaGetLastError());
    TERM_CHECK(cudaMemcpy(out_grad, dg.p, kTermParams * 4, cudaMemcpyDeviceToHost));
    TERM_CHECK(cudaMemcpy(out_loss, dl.p, 4, cudaMemcpyDeviceToHost));
    return cudaSuccess;
}

cudaError_t term_train(const float* feats, const float* labels, uint64_t n, float* params, uint32_t epochs,
                       uint32_t batch, float lr, float pos_weight, float weight_decay, uint64_t seed,
                       float* out_epoch_loss) {
    if (batch == 0) batch = 1024;
    const uint64_t max_tiles = (std::min<uint64_t>(batch, n) + kTile - 1) / kTile;
    const uint64_t nb = (n + batch - 1) / batch;
    const uint64_t nep = std::max<uint32_t>(epochs, 1);
    // one allocation: each takes about 0.4 ms, and as much to free
    DevArray<float> ws;
    const uint64_t sizes[] = {kTermParams, kTermParams, kTermParams, nep, 2, max_tiles * kTermParams, max_tiles,
                              2 * nb, n, n, n * kTermFeatures};
    constexpr int kParts = sizeof(sizes) / sizeof(sizes[0]);
    float* at[kParts];
    uint64_t total = 0;
    for (int i = 0; i < kParts; i++) total += (sizes[i] + 63) / 64 * 64;
    TERM_CHECK(ws.alloc(total));
    total = 0;
    for (int i = 0; i < kParts; i++) {
        at[i] = ws.p + total;
        total += (sizes[i] + 63) / 64 * 64;
    }
    TrainArgs a{};
    a.params = at[0];
    a.m = at[1];
    a.v = at[2];
    a.barrier = reinterpret_cast<uint32_t*>(at[4]);
    a.failed = a.barrier + 1;
    a.part = at[5];
    a.part_loss = at[6];
    a.bias = reinterpret_cast<const float2*>(at[7]);
    a.labels = at[8];
    a.perm = reinterpret_cast<const uint32_t*>(at[9]);
    a.feats = at[10];
    a.n = n;
    a.batch = batch;
    a.lr = lr;
    a.pos_weight = pos_weight;
    a.wd = weight_decay;
    TERM_CHECK(cudaMemset(a.m, 0, (size_t)(a.part - a.m) * 4));  // moments, epoch losses, barrier
    TERM_CHECK(cudaMemcpy(a.params, params, kTermParams * 4, cudaMemcpyHostToDevice));
    TERM_CHECK(cudaMemcpy(at[10], feats, n * kTermFeatures * 4, cudaMemcpyHostToDevice));
    TERM_CHECK(cudaMemcpy(at[8], labels, n * 4, cudaMemcpyHostToDevice));
    const int smem = (int)sizeof(TrainSmem);
    TERM_CHECK(cudaFuncSetAttribute(term_epoch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int dev = 0, sms = 0, per_sm = 0;
    TERM_CHECK(cudaGetDevice(&dev));
    TERM_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TERM_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, term_epoch_kernel, kGradThreads, smem));
    const unsigned grid = (unsigned)std::min<uint64_t>(max_tiles * kSplit, (uint64_t)sms * (uint64_t)std::max(per_sm, 1));
    std::vector<uint32_t> perm(n);
    std::iota(perm.begin(), perm.end(), 0u);
    std::mt19937_64 rng(seed);
    std::vector<float2> bias(nb);
    uint64_t step = 0;
    if (epochs) std::shuffle(perm.begin(), perm.end(), rng);
    for (uint32_t ep = 0; ep < epochs; ep++) {
        for (uint64_t b = 0; b < nb; b++) {
            step++;
            bias[b] = make_float2(1.f - (float)std::pow(0.9, (double)step), 1.f - (float)std::pow(0.999, (double)step));
        }
        // (these copies wait for the last epoch)
        TERM_CHECK(cudaMemcpy(at[9], perm.data(), n * 4, cudaMemcpyHostToDevice));
        TERM_CHECK(cudaMemcpy(at[7], bias.data(), nb * sizeof(float2), cudaMemcpyHostToDevice));
        a.epoch_loss = at[3] + ep;
        a.gen = (uint32_t)(2 * nb * ep);
        void* args[] = {&a};
        TERM_CHECK(cudaLaunchCooperativeKernel((const void*)term_epoch_kernel, dim3(grid), dim3(kGradThreads), args, (size_t)smem, 0));
        // the next epoch's order, while this one runs
        if (ep + 1 < epochs) std::shuffle(perm.begin(), perm.end(), rng);
    }
    uint32_t failed = 0;
    TERM_CHECK(cudaMemcpy(&failed, a.failed, 4, cudaMemcpyDeviceToHost));
    if (failed) return cudaErrorLaunchTimeout;
    if (out_epoch_loss && epochs) {
        TERM_CHECK(cudaMemcpy(out_epoch_loss, at[3], epochs * 4, cudaMemcpyDeviceToHost));
        for (uint32_t ep = 0; ep < epochs; ep++) out_epoch_loss[ep] = nb ? out_epoch_loss[ep] / (float)nb : 0.f;
    }
    TERM_CHECK(cudaMemcpy(params, a.params, kTermParams * 4, cudaMemcpyDeviceToHost));
    return cudaSuccess;
}

cudaError_t term_logits(const float* params, const float* feats, uint64_t n, float* out) {
    std::vector<unsigned char> packed(kTermPackedBytes);
    pack_term_model(params, packed.data());
    DevArray<unsigned char> dmodel;
    DevArray<float> df, dout;
    TERM_CHECK(dmodel.alloc(kTermPackedBytes));
    TERM_CHECK(df.alloc(n * kTermFeatures));
    TERM_CHECK(dout.alloc(n));
    TERM_CHECK(cudaMemcpy(dmodel.p, packed.data(), kTermPackedBytes, cudaMemcpyHostToDevice));
    TERM_CHECK(cudaMemcpy(df.p, feats, n * kTermFeatures * 4, cudaMemcpyHostToDevice));
    if (n) {
        term_logits_kernel<<<(unsigned)((n + 7) / 8), 256>>>(reinterpret_cast<const float*>(dmodel.p), df.p, n, dout.p);
        TERM_CHECK(cudaGetLastError());
    }
    TERM_CHECK(cudaMemcpy(out, dout.p, n * 4, cudaMemcpyDeviceToHost));
    return cudaSuccess;
}

}  // namespace hnswgpu
