// Offsets from sums over blocks of items: a counting pass adds each item's
// two counts to its block's 64-bit sum (the first in the low half), the
// blocks' sums are scanned here, and a second pass over the blocks that hold
// anything turns them into the items' offsets.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace iso {
namespace {

constexpr unsigned long long NO_ITEMS = ~0ull;  // the scanned sum of a block that holds nothing

// Exclusive scan in place by one thread block, four entries per thread and
// turn; totals: both grand totals.
__global__ void __launch_bounds__(1024) scan_block_sums(unsigned long long* sums, uint32_t nblocks, uint2* totals) {
    __shared__ unsigned long long part[32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (uint32_t b0 = 0; b0 < nblocks; b0 += 4096) {
        const uint32_t at = b0 + 4 * threadIdx.x;
        unsigned long long v[4], mine = 0;
        for (uint32_t k = 0; k < 4; ++k) {
            v[k] = at + k < nblocks ? sums[at + k] : 0;
            mine += v[k];
        }
        unsigned long long incl = mine;
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) part[w] = incl;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (uint32_t k = 0; k < 32; ++k) {
            if (k < w) before += part[k];
            all += part[k];
        }
        unsigned long long run = carry + before + incl - mine;
        for (uint32_t k = 0; k < 4; ++k) {
            if (at + k < nblocks) sums[at + k] = v[k] ? run : NO_ITEMS;
            run += v[k];
        }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *totals = make_uint2((uint32_t)carry, (uint32_t)(carry >> 32));
}

// The offset of a thread's own items, `mine` their sum, in a block of 256
// threads that holds the scanned sum `base` (every thread calls it once).
__device__ __forceinline__ unsigned long long offset_in_block(unsigned long long base, unsigned long long mine) {
    __shared__ unsigned long long part[8];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long incl = mine;
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) part[w] = incl;
    __syncthreads();
    unsigned long long run = base + incl - mine;
    for (uint32_t k = 0; k < w; ++k) run += part[k];
    return run;
}

}  // namespace
}  // namespace iso
