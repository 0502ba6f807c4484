// tt_rank_groups.h — how the spanning forest's edges join (tt_dim0.cu).
//
// The forest's rounds take the m sorted edges of n vertices in groups, one a
// host round trip: the edges [end[t - 1], end[t]) join in trip t, and after the
// third trip nothing is left to join. The kernels walk a group as a range of
// ranks, so the ends never fall and the last is m.
#pragma once
#include <cstdint>

namespace tt {

struct RankGroups {
    uint64_t end[3];
};

// Groups of 8 n, then 64 n edges, then the rest. With fewer than 16 n edges (kNN
// graphs), or fewer than 2^17 in all, the extra trips would cost more than the
// passes they save, and all join at once.
inline RankGroups rank_groups(uint64_t m, uint64_t n) {
    if (m < 16 * n || m < (uint64_t(1) << 17)) return RankGroups{{m, m, m}};
    return RankGroups{{8 * n, m < 72 * n ? m : 72 * n, m}};
}

}  // namespace tt
