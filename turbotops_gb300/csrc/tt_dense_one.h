// tt_dense_one.h — which clouds take one block for their matrix and radius
// (tt_dense.cu k_dense_one).
#pragma once
#include <cstdint>

namespace tt {

constexpr uint32_t kOneN = 128;
constexpr uint32_t kOneLpN = 91;         // Lp (see dense_one_block)
constexpr uint32_t kOneFloats = 12000;   // floats that 48 KB hold beside the row maxima

// A point's floats in shared memory: an odd number, so that a warp's points
// start in different banks.
inline uint32_t dense_one_stride(uint32_t dim) { return dim | 1u; }

// Up to 128 points: two memsets, two kernels and a copy take 30 us, the block
// 13 to 32 us up to 32 coordinates (128 points: R^3 22, R^32 32; with the points
// dim floats apart R^32 150), 50 at 93 (the kernels 93). Lp is bound by
// arithmetic, one SM's share of it: 91 points in R^3 131 us (the kernels 142), 128
// points 247 (142). (Floats in 64 bits: 128 points of 2^25 coordinates are 2^32.)
inline bool dense_one_block(uint32_t n, uint32_t dim, bool lp) {
    return n <= (lp ? kOneLpN : kOneN) && uint64_t(n) * dense_one_stride(dim) <= kOneFloats;
}

}  // namespace tt
