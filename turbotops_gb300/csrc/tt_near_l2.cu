// tt_near_l2.cu — the ordered searches (tt_near.cuh) for L2.
#define TT_NEAR_IMPL
#include <cmath>
#include <type_traits>

#include "tt_near.cuh"

namespace tt {
namespace near {
TT_NEAR_INSTANTIATE(M_L2)
}  // namespace near
}  // namespace tt
