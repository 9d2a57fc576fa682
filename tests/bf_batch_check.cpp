// The exact scan's choice of how many queries share its workspace
// (bf_search.h) against an allocator that has little memory: every amount that
// holds one query's keys is enough.  Prints "ok" or the first failure.
#include <cstdint>
#include <cstdio>

#include "bf_search.h"

using namespace hnswgpu;

int main() {
    for (uint32_t start : {1u, 2u, 3u, 7u, 8u, 9u, 40u, 1000u})
        for (uint32_t room = 0; room <= 1100; room++) {
            uint32_t batch = start, last = 0;
            const cudaError_t e = bf_fit_batch(batch, [&](uint32_t b) {
                last = b;
                return b <= room ? cudaSuccess : cudaErrorMemoryAllocation;
            });
            const bool ok = room == 0 ? e == cudaErrorMemoryAllocation
                                      : e == cudaSuccess && batch == last && batch >= 1 && batch <= start && batch <= room;
            if (!ok) {
                std::printf("start %u room %u: error %d batch %u\n", start, room, (int)e, batch);
                return 1;
            }
        }
    // another error is not retried
    uint32_t batch = 8, calls = 0;
    if (bf_fit_batch(batch, [&](uint32_t) { calls++; return cudaErrorInvalidValue; }) != cudaErrorInvalidValue || calls != 1) return 1;
    std::printf("ok\n");
    return 0;
}
