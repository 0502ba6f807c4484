// tt_dense_one.h — which clouds take one block for their matrix and radius
// (tt_dense.cu k_dense_one).
#pragma once
#include <cstdint>

namespace tt {

constexpr uint32_t kOneN = 128;
constexpr uint32_t kOneFloats = 12000;   // points x dim that 48 KB hold beside the row maxima

// (in 64 bits: 128 points of 2^25 coordinates are 2^32 floats)
inline bool dense_one_block(uint32_t n, uint32_t dim) { return n <= kOneN && uint64_t(n) * dim <= kOneFloats; }

}  // namespace tt
