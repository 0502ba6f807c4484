// tt_near_graph_l2.cu — the ordered radius rows and foreign searches
// (tt_near.cuh) for L2.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void near_foreign<M_L2>(tt_ctx*, const View&, u32, const u32*, const u32*, const u32*, const u32*, const u32*,
                                u32*, unsigned long long*);
template void near_radius_count<M_L2>(tt_ctx*, const View&, u32, f32, u64*, u32*);
template void near_radius_fill<M_L2>(tt_ctx*, const View&, u32, f32, u32, const u64*, u32*, f32*);
}  // namespace near
}  // namespace tt
