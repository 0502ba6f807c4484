// tt_near_l1.cu — the ordered kNN lists (tt_near.cuh) for L1.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void near_knn<M_L1>(tt_ctx*, const View&, u32, u32, u32*, f32*);
}  // namespace near
}  // namespace tt
