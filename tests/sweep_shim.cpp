// sweep_shim.cpp — test harness only: the product's compute_pairs on one dense
// complex with its edges in order (sweeps, cocycles) beside the same without,
// compiled with the host compiler.
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../turbotops_gb300/csrc/tt_reduce.h"

// 1: the same bars (values, order, critical simplices), pivots and counts; 0: they
// differ. *asked: whether the edges were asked for; *emergent: the emergent pairs.
extern "C" int sweeps_agree(const float* mat, uint32_t n, float thr, const uint64_t* cidx, const float* cd,
                            uint64_t ncols, const uint64_t* emi, const uint8_t* emf, uint64_t patience,
                            unsigned threads, uint32_t* asked, uint64_t* emergent) {
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
    *asked = 0;
    const SortedEdges edges{[&] {
                                ++*asked;
                                return keys.data();
                            },
                            keys.size(), patience};
    const Bars x = compute_pairs(hc, 1, 1, cols, emi, emf, p, s, threads, &edges);
    const Bars y = compute_pairs(hc, 1, 1, cols, emi, emf, q, t, 1);
    *emergent = t.emergent;
    return x.birth == y.birth && x.death == y.death && x.birth_idx == y.birth_idx && x.death_idx == y.death_idx &&
           p == q && s.columns == t.columns && s.emergent == t.emergent && *asked <= 1;
}
