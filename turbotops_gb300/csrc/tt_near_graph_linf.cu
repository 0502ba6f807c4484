// tt_near_graph_linf.cu — the ordered radius rows and foreign searches
// (tt_near.cuh) for Linf.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {
template void near_foreign<M_LINF>(tt_ctx*, const View&, u32, const u32*, const u32*, const u32*, const u32*, const u32*,
                                u32*, unsigned long long*);
template void near_radius_count<M_LINF>(tt_ctx*, const View&, u32, f32, u64*, u32*);
template void near_radius_fill<M_LINF>(tt_ctx*, const View&, u32, f32, u32, const u64*, u32*, f32*);
}  // namespace near
}  // namespace tt
