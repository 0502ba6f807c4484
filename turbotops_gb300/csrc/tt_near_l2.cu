// tt_near_l2.cu — the ordered kNN lists (tt_near.cuh) for L2.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void near_knn<M_L2>(tt_ctx*, const View&, u32, u32, u32*, f32*);
}  // namespace near
}  // namespace tt
