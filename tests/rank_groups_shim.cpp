// rank_groups_shim.cpp — test harness only: the forest's rank groups, compiled
// with the host compiler.
#include "../turbotops_gb300/csrc/tt_rank_groups.h"

extern "C" void rank_groups(uint64_t m, uint64_t n, uint64_t* end) {
    const tt::RankGroups g = tt::rank_groups(m, n);
    for (int t = 0; t < 3; ++t) end[t] = g.end[t];
}
