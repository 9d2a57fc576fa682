// Launch parameters of the brute-force search kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace hnswgpu {

struct BfParams {
    const float* vecs;       // count x row_floats, zero padded
    const uint64_t* labels;  // count
    const uint8_t* allow;    // optional mask over row ids
    uint32_t count, dim, row_floats;
    const float* queries;    // nq x dim
    uint32_t nq, k, normalize;
    uint64_t* out_labels;
    float* out_dists;
    int32_t* out_counts;
    // workspace of one batch of queries (set by launch_bf_search)
    uint32_t* keys;          // nq x count distance keys
    uint32_t* gmin;          // nq x groups: smallest allowed key of 32 rows
    uint32_t groups;         // ceil(count / 32)
};

// Whether k results over rows of row_floats floats are within the interface's limits.
bool bf_supported(uint32_t k, uint32_t row_floats, size_t max_smem);
// Queries of p that run at once, and the bytes of workspace for `batch` at once.
uint32_t bf_batch(const BfParams& p);
size_t bf_workspace(const BfParams& p, uint32_t batch);
// Allocates for `batch` queries at once, fewer where memory is short: down to
// one, whose keys are the least the scan can do with.
template <class Alloc>
cudaError_t bf_fit_batch(uint32_t& batch, Alloc alloc) {
    cudaError_t e = alloc(batch);
    while (e == cudaErrorMemoryAllocation && batch > 1) {
        batch = batch / 4 > 1 ? batch / 4 : 1;
        e = alloc(batch);
    }
    return e;
}
cudaError_t launch_bf_search(BfParams p, int space, void* workspace, uint32_t batch, cudaStream_t stream);

}  // namespace hnswgpu
