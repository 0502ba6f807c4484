// tt_near_lp.cu — the ordered kNN lists (tt_near.cuh) for Lp: any exponent's
// kernels, and the choice of the class.
#define TT_NEAR_IMPL
#include "tt_near.cuh"

namespace tt {
namespace near {

extern template void knn_lp_class<1>(tt_ctx*, const View&, u32, u32, u32*, f32*);
extern template void knn_lp_class<2>(tt_ctx*, const View&, u32, u32, u32*, f32*);

void near_knn_lp(tt_ctx* c, View v, u32 dim, f32 p, u32 k, u32* ids, f32* dists) {
    v.p = p;
    switch (pow_class(p)) {
        case 1: knn_lp_class<1>(c, v, dim, k, ids, dists); break;
        case 2: knn_lp_class<2>(c, v, dim, k, ids, dists); break;
        default: knn_lp_class<0>(c, v, dim, k, ids, dists); break;
    }
}

}  // namespace near
}  // namespace tt
