// tt_warp_sort.cuh — a warp's keys ordered in registers.
#pragma once
#include "tt_common.cuh"

namespace tt {

// K keys a lane, ascending over (lane, key). Each merge of two ascending runs
// compares mirrored keys first, so that every later step keeps the smaller key
// in the lower place.
template <int K>
__device__ __forceinline__ void sort_lane_keys(u32 (&key)[K]) {
    const u32 lane = threadIdx.x & 31;
    auto order = [&](int i, int j) {
        const u32 x = key[i], y = key[j];
        key[i] = min(x, y);
        key[j] = max(x, y);
    };
#pragma unroll
    for (int size = 2; size <= K; size <<= 1) {
#pragma unroll
        for (int i = 0; i < K; ++i)
            if ((i & (size >> 1)) == 0) order(i, i ^ (size - 1));
#pragma unroll
        for (int stride = size >> 2; stride; stride >>= 1)
#pragma unroll
            for (int i = 0; i < K; ++i)
                if ((i & stride) == 0) order(i, i | stride);
    }
#pragma unroll 1
    for (u32 size = 2; size <= 32; size <<= 1) {   // runs of size lanes
        {
            const bool low = (lane & (size >> 1)) == 0;
#pragma unroll
            for (int i = 0; i < (K + 1) / 2; ++i) {
                const u32 x = __shfl_xor_sync(0xffffffffu, key[K - 1 - i], size - 1);
                const u32 y = __shfl_xor_sync(0xffffffffu, key[i], size - 1);
                key[i] = low ? min(key[i], x) : max(key[i], x);
                if (K > 1) key[K - 1 - i] = low ? min(key[K - 1 - i], y) : max(key[K - 1 - i], y);
            }
        }
#pragma unroll 1
        for (u32 stride = size >> 2; stride; stride >>= 1) {
            const bool low = (lane & stride) == 0;
#pragma unroll
            for (int i = 0; i < K; ++i) {
                const u32 x = __shfl_xor_sync(0xffffffffu, key[i], stride);
                key[i] = low ? min(key[i], x) : max(key[i], x);
            }
        }
#pragma unroll
        for (int stride = K >> 1; stride; stride >>= 1)
#pragma unroll
            for (int i = 0; i < K; ++i)
                if ((i & stride) == 0) order(i, i | stride);
    }
}

}  // namespace tt
