// tt_near_lp.cu — the ordered searches (tt_near.cuh) for Lp.
#define TT_NEAR_IMPL
#include <cmath>
#include <type_traits>

#include "tt_near.cuh"

namespace tt {
namespace near {

template <int CLS>
static void run(tt_ctx* c, const View& v, u32 dim, u32 k, u32* ids, f32* dists) {
    constexpr int KIND = M_LP + 16 * CLS;
    with_dim<KIND>(dim, [&](auto dp, auto) {
        constexpr int DP = decltype(dp)::value, QW = queries_per_warp(DP);
        launch_pdl(k_near_knn_lp<KIND, DP, QW>, div_up(div_up(v.n, QW), kWarps), 32 * kWarps, 0, c->stream, v, dim, k,
                   ids, dists);
        TT_LAUNCH("k_near_knn_lp");
        ++c->launches;
    });
}

void near_knn_lp(tt_ctx* c, View v, u32 dim, f32 p, u32 k, u32* ids, f32* dists) {
    v.p = p;
    switch (pow_class(p)) {
        case 1: run<1>(c, v, dim, k, ids, dists); break;
        case 2: run<2>(c, v, dim, k, ids, dists); break;
        default: run<0>(c, v, dim, k, ids, dists); break;
    }
}

}  // namespace near
}  // namespace tt
