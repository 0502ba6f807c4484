// tt_near_linf.cu — the ordered searches (tt_near.cuh) for Linf.
#define TT_NEAR_IMPL
#include <cmath>
#include <type_traits>

#include "tt_near.cuh"

namespace tt {
namespace near {
TT_NEAR_INSTANTIATE(M_LINF)
}  // namespace near
}  // namespace tt
