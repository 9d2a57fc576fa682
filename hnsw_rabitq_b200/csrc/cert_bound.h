// How far a bf16 tensor-core distance may lie from the reference's float32
// distance of the same query and row (bf_tc.cu's certificate).  Usable from host
// code for testing.
#pragma once
#include <cstdint>

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#endif

namespace hnswgpu {

// Loss of one MMA step (16 products and the accumulator) in units of 2^-23 of
// |q'||x'|, which bounds every product and partial sum.  How the tensor cores
// add is not documented, so this is an assumption with a margin: groups of at
// least four products and the accumulator, each addend aligned to the largest
// and cut at 24 bits.  A group of g then loses at most (g + 1) 2^-23 in its
// addends and 2^-23 in its sum, 16 / g times a step: 24 for g = 4, fewer for
// larger ones.  Library bf16 GEMMs of such inputs (768 dims) are off by 1.5e-6 of
// |q||x|, where this allows 1.4e-4.
constexpr double kMmaLoss = 24.0;

// space 0: squared L2, 1: inner product.  nq, M: norms of the query and of the
// longest row; dq, D: norms of their rounding errors (q' and x' are the rounded
// ones).  |q.x - q'.x'| <= |q - q'||x| + |q'||x - x'| (Cauchy-Schwarz), the MMA
// steps over rows padded to 64, and the float32 arithmetic of the reference's
// summation and of the norms, at most dim / 4 + 64 roundings of 2^-24: twice
// that.  Subnormal inputs the tensor cores may drop: the 2^-126 term.
__host__ __device__ inline double cert_bound(int space, uint32_t dim, double nq, double dq, double M, double D) {
    const double eps = 1.0 / (1 << 23);
    const double steps = (double)((dim + 63) / 64 * 4);
    const double E = dq * M + (nq + dq) * D + steps * kMmaLoss * eps * (nq + dq) * (M + D) +
                     (nq + M + 1.0) * dim * 1.2e-38;
    const double g = (dim / 4 + 64) * eps;
    return space == 0 ? 2.0 * E + g * (nq + M) * (nq + M) : E + g * nq * M + 2.0 * eps * (1.0 + nq * M);
}

}  // namespace hnswgpu
