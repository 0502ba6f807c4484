// cocycle_shim.cpp — test harness only: the product's dense_pairs_dim1 beside its
// compute_pairs on one dense complex, compiled with the host compiler.
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../turbotops_gb300/csrc/tt_reduce.h"

// 1: the same bars (values, order, critical simplices) and pivots; 0: they
// differ; 2: dense_pairs_dim1 declined. *bars: how many.
extern "C" int cocycles_agree(const float* mat, uint32_t n, float thr, const uint64_t* cidx, const float* cd,
                              uint64_t ncols, uint64_t budget, uint64_t* bars) {
    using namespace tt::host;
    const HostComplex hc{mat, nullptr, nullptr, nullptr, n, thr};
    std::vector<Entry> cols(ncols);
    for (uint64_t i = 0; i < ncols; ++i) cols[i] = Entry{cidx[i], cd[i]};
    std::vector<uint64_t> keys;
    for (uint64_t a = 1; a < n; ++a)
        for (uint64_t b = 0; b < a; ++b) {
            const float d = mat[a * n + b];
            if (!(d <= thr)) continue;
            uint32_t u;
            std::memcpy(&u, &d, 4);
            keys.push_back((uint64_t(u) << 33) | (((uint64_t(1) << 33) - 1) - (a * (a - 1) / 2 + b)));
        }
    std::sort(keys.begin(), keys.end());
    std::vector<uint64_t> p, q;
    ReduceStats s, t;
    Bars x;
    if (!dense_pairs_dim1(hc, cols, keys.data(), keys.size(), x, p, s, budget)) return 2;
    const Bars y = compute_pairs(hc, 1, 1, cols, nullptr, nullptr, q, t, 1);
    *bars = x.birth.size();
    return x.birth == y.birth && x.death == y.death && x.birth_idx == y.birth_idx && x.death_idx == y.death_idx && p == q;
}
