// tt_near_linf.cu — the ordered kNN lists (tt_near.cuh) for Linf.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void near_knn<M_LINF>(tt_ctx*, const View&, u32, u32, u32*, f32*);
}  // namespace near
}  // namespace tt
