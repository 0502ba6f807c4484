// tt_near_l1.cu — the ordered searches (tt_near.cuh) for L1.
#define TT_NEAR_IMPL
#include <cmath>
#include <type_traits>

#include "tt_near.cuh"

namespace tt {
namespace near {
TT_NEAR_INSTANTIATE(M_L1)
}  // namespace near
}  // namespace tt
