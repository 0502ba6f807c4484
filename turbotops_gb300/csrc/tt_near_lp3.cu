// tt_near_lp3.cu — the ordered kNN lists (tt_near.cuh) for exponent 3.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void knn_lp_class<2>(tt_ctx*, const View&, u32, u32, u32*, f32*);
}  // namespace near
}  // namespace tt
