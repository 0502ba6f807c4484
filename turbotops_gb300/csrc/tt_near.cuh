// tt_near.cuh — exact all-pairs searches over points in a spatial order: the
// same results as the exhaustive scans of tt_scan.cuh (which replace
// graph.hpp knn_lists_exact :211-225 and radius_graph :170-201), reading only
// the tiles of points whose bounding box can hold an answer.
//
// Order (tt_near.cu). The points are sorted so that 32 consecutive ones (a
// tile) are close together; every tile, and every 32 tiles (a super tile),
// keeps its bounding box. The coordinates are regrouped tile by tile,
// coordinate-major, so that a warp reads a tile with one coalesced load a
// coordinate: lane = candidate.
//
// Search. A warp owns QW consecutive queries of the order. It tests 32 super
// tiles at a time, then the 32 tiles of the super tile, one a lane, always
// going on with the closest box, and stops where the closest one is farther
// than every query's current bound. The candidates of a tile are held in
// registers and tested against the queries that still need it, in turn (their
// coordinates broadcast from shared memory), so more queries a warp reuse the
// tile's loads: 1 up to four dimensions, 8 from 32 on. Every query is tested
// against every box on its own (a common box of 8 points in R^32 reaches into
// every cluster: 100,000 mixture points' foreign searches took 70 ms with it).
//
// Why no result changes. The lower bound of a box is the metric's own
// lane-ordered float evaluation (tt_metric.cuh) of the gap vector
// max(lo - q, q - hi, 0): every step (subtract, fma of a square, add of an
// absolute value, max) is monotone under round-to-nearest, and every
// candidate's |q - c| is at least the gap coordinate by coordinate, so the
// bound is at most the computed distance of every point in the box, bit for
// bit, with no margin. A box is skipped only when its bound exceeds the
// query's bound strictly, the same test that drops a candidate, and all lists
// compare (distance, id), so the visiting order does not matter.
// Coordinates padded with zeros beyond the dimension add exact zeros to the
// sums, in the same lane order. Lp's own evaluation is long (a power series a
// coordinate, a root in double precision) and not monotone in its last bits:
// there boxes and candidates are tested on a fast power sum with a margin for
// every error (below, k_near_knn_lp), and only the survivors are evaluated.
#pragma once
#include <cmath>
#include <type_traits>

#include "tt_internal.cuh"
#include "tt_metric.cuh"
#include "tt_warp_sort.cuh"

namespace tt {
namespace near {

constexpr u32 kTile = 32;
constexpr u32 kWarps = 4;          // warps a block
constexpr u32 kMaxDim = 64;
constexpr u32 kProjectDim = 16;    // padded dimensions from which tiles are also tested along a direction

// The points in order. Boxes: lower corners, then upper ones, coordinate by
// coordinate (row k: the tiles' values, padded to `tpad` / `spad` columns).
struct View {
    const f32* xt = nullptr;   // [ntiles][dp][32]
    const u32* id = nullptr;   // [ntiles * 32]: original ids, ~0 past n
    const f32* tbox = nullptr;   // [2 * dp][tpad]
    const f32* sbox = nullptr;   // [2 * dp][spad]
    const f32* abox = nullptr;   // [ntiles][2][dp]: the tiles' corners again (dp >= kProjectDim; else null)
    const f32* sep = nullptr;    // [nblk][nblk]: lower bounds between blocks of 4 tiles (near_separations; or null)
    u32 nblk = 0;
    u32 n = 0, ntiles = 0, nsup = 0, tpad = 0, spad = 0;
    f32 p = 2.0f;    // Lp: the exponent
};

// Coordinates held for `dim` (zero-padded) and 16-coordinate chunks in the
// metric's lane order (l2_sq_acc, l1_acc: dim / 16; linf is order-free).
inline u32 padded_dim(u32 dim) {
    return dim <= 4 ? (dim < 2 ? 2 : dim) : dim <= 8 ? 8 : dim <= 16 ? 16 : dim <= 32 ? 32 : dim <= 48 ? 48 : 64;
}

// Queries a warp takes at once (tt_near.cuh's header).
constexpr u32 queries_per_warp(u32 dp) { return dp <= 4 ? 1 : dp <= 8 ? 2 : dp <= 16 ? 4 : 8; }
constexpr u32 kFewPoints = 10000;   // lists of fewer points: half as many queries a warp (launch_knn)

// tt_near.cu
constexpr u32 kBlockTiles = 4;          // tiles a separation block
constexpr u32 kSepMaxBlocks = 4096;     // 64 MB of separations, 201 with the sums they are made from
constexpr u32 kSepMinPoints = 2048;
// Fills v.sep for the metric where it pays (kProjectDim, L1, L2, Lp).
void near_separations(tt_ctx* c, View& v, u32 dim, int kind, f32 p);
View near_order(tt_ctx* c, const f32* x, u32 n, u32 dim);
View near_regroup(tt_ctx* c, const f32* x, u32 n, u32 dim, const u32* perm);   // in a given order

// tt_near_*.cu (kernels by metric, several translation units so that they
// compile in parallel)
template <int KIND>
void near_knn(tt_ctx* c, const View& v, u32 dim, u32 k, u32* ids, f32* dists);
// (*longest: the longest row, where one is longer than kRadiusRow / 2)
template <int KIND>
void near_radius_count(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest);
template <int KIND>
void near_radius_fill(tt_ctx* c, const View& v, u32 dim, f32 tau, u32 longest, const u64* rp, u32* ci, f32* w);
void near_knn_lp(tt_ctx* c, View v, u32 dim, f32 p, u32 k, u32* ids, f32* dists);   // p <= kLpMax
constexpr f32 kLpMax = 64.0f;
constexpr u32 kRadiusRow = 1024;   // longest row the fill sorts
// One round's proposals of the listed queries (k_near_foreign).
template <int KIND>
void near_foreign(tt_ctx* c, const View& v, u32 dim, const u32* cpos, const u32* tcomp, const u32* scomp,
                  const u32* qlist, const u32* nq, u32* bd, unsigned long long* near);
// Components in the points' order: cpos[position], and the component a tile
// or a super tile shares (tt_near.cu).
void near_components(tt_ctx* c, const View& v, const u32* comp, u32* cpos, u32* tcomp, u32* scomp);
// The queries of a round, listed by position in whole groups of
// queries_per_warp (~0 fills a group up), *nq the list's length: the points
// without a proposal whose kb (K-th neighbour's distance bits; null: every
// point) does not exceed their component's best so far.
void near_queries(tt_ctx* c, const View& v, u32 dim, const u32* cpos, const unsigned long long* near, const u32* kb,
                  const u32* bd, u32* qlist, u32* nq);

#ifdef TT_NEAR_IMPL

// |d|^p, fast: exp2(p log2 |d|) on the special-function unit, or, for the two
// exponents below, the product (cls 1: 1.5; cls 2: 3). Others have a short product
// too (2.5, 4), but every class is one more copy of the kernels for all
// dimensions, a fifth of the library's build; these two are the ones that the
// workloads here and the tests use, and the rest take the general form (100,000 x
// 32 mixture points, k = 15: L1.5 7.1 ms,
// L3 6.0, by the general form 9.2). 0 and subnormal
// |d| give 0, NaN stays NaN.
__device__ __forceinline__ f32 sqrt_fast(f32 x) {
    f32 r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <int CLS>
__device__ __forceinline__ f32 pow_abs(f32 d, f32 p) {
    const f32 a = fabsf(d);
    if constexpr (CLS == 1) return a * sqrt_fast(a);                // 1.5
    else if constexpr (CLS == 2) return a * a * a;                  // 3
    else {
        f32 l, r;
        asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(a));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(p * l));
        return r;
    }
}
inline int pow_class(f32 p) { return p == 1.5f ? 1 : p == 3.0f ? 2 : 0; }
// The kernels' kind for Lp names the class too: M_LP + 16 cls (a class for
// each kernel: with a switch at every power the code outgrew the instruction
// cache, and a fetch stall took 40 % of the cycles).
constexpr bool is_lp(int kind) { return (kind & 15) == M_LP; }
template <int KIND, int DP, typename Diff>
__device__ __forceinline__ f32 pow_sum(const Diff& diff, f32 p) {
    f32 t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < DP; ++k) t[k & 3] += pow_abs<(KIND >> 4)>(diff(k), p);
    return (t[0] + t[1]) + (t[2] + t[3]);
}

// The metric's evaluation before its final root (L2: the squared sum), of
// d[k] = q[k] - c[k], the query's coordinates in shared memory, the
// candidate's (or the gap's) in registers; the lane order of tt_metric.cuh
// for dim coordinates with CH = dim / 16 chunks, zero-padded to DP.
template <int KIND, int DP, int CH, typename Diff>
__device__ __forceinline__ f32 eval(const Diff& diff, f32 p = 2.0f) {
    if constexpr (is_lp(KIND)) {
        return pow_sum<KIND, DP>(diff, p);
    } else if constexpr (KIND == M_LINF) {
        f32 m = 0.0f;
#pragma unroll
        for (int k = 0; k < DP; ++k) m = fmaxf(m, fabsf(diff(k)));
        return m;
    } else {
        auto term = [&](int k, f32 s) -> f32 {
            const f32 d = diff(k);
            if constexpr (KIND == M_L2) return __fmaf_rn(d, d, s);
            else return __fadd_rn(s, fabsf(d));
        };
        f32 s = 0.0f;
        if constexpr (CH > 0) {
            f32 t[8];
#pragma unroll
            for (int l = 0; l < 8; ++l) {
                f32 a0 = 0.0f, a1 = 0.0f;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    a0 = term(16 * c + l, a0);
                    a1 = term(16 * c + 8 + l, a1);
                }
                t[l] = __fadd_rn(a0, a1);
            }
            s = hsum8(t);
        }
#pragma unroll
        for (int k = 16 * CH; k < DP; ++k) s = term(k, s);
        return s;
    }
}

// The query bound that eval's values are compared with, from a distance.
template <int KIND>
__device__ __forceinline__ f32 bound_of(f32 d) {
    if constexpr (KIND == M_L2) return sq_bound(d);
    else return d;
}

// A distance that every point whose computed distance is at most d lies
// within: the evaluations err by less than 2^-15 (L1, L2: 66 roundings of
// 2^-24; Lp: k_near_knn_lp).
__device__ __forceinline__ f32 bound_margin(f32 d) { return d * (1.0f + 0x1p-10f); }

template <int DP>
constexpr int row_floats() { return (DP + 3) / 4 * 4; }

// One warp's queries: coordinates, common box, bounds.
template <int DP, int QW>
struct WarpQ {
    alignas(16) f32 q[QW][row_floats<DP>()];
    alignas(16) f32 qt[DP][QW];   // the same, coordinate-major
    f32 thr[QW];   // eval values above it cannot matter (negative: no query)
    f32 bnd[QW];   // distances above it cannot matter (bound_margin)
    u32 blk[QW];   // its separation block
    u32 own[QW];
};

// The queries that box column t may matter to (a bit each), and the smallest
// of their lower bounds in b (float bits; ~0: none). One query: its bound is
// the metric's lane-ordered evaluation of the gaps. More: the sums run over
// the coordinates for all queries at once (a box's corners are read once),
// rounded down, and the margin 2^-16 covers the candidate sums' own rounding
// (at most 66 operations, each within 2^-24).
template <int KIND, int DP, int CH, int QW>
__device__ __forceinline__ u32 box_needs(const f32* __restrict__ box, u32 pad, u32 t, const WarpQ<DP, QW>& W, f32 p,
                                         u32& b) {
    // (infinities that cancel leave a NaN, which fmaxf drops: a gap of 0)
    auto gap = [](f32 lo, f32 hi, f32 q) -> f32 { return fmaxf(fmaxf(__fsub_rn(lo, q), __fsub_rn(q, hi)), 0.0f); };
    if constexpr (QW == 1) {
        const f32 s = eval<KIND, DP, CH>(
            [&](int k) -> f32 { return gap(__ldg(box + u64(k) * pad + t), __ldg(box + u64(DP + k) * pad + t), W.qt[k][0]); },
            p);
        b = __float_as_uint(s);
        if (!(s > W.thr[0])) return 1u;
        b = 0xffffffffu;
        return 0u;
    } else {
        f32 s[QW];
#pragma unroll
        for (int q = 0; q < QW; ++q) s[q] = 0.0f;
        auto add = [&](auto&& term) {
#pragma unroll 4
            for (int k = 0; k < DP; ++k) {
                const f32 lo = __ldg(box + u64(k) * pad + t), hi = __ldg(box + u64(DP + k) * pad + t);
#pragma unroll
                for (int q = 0; q < QW; ++q) s[q] = term(gap(lo, hi, W.qt[k][q]), s[q]);
            }
        };
        if constexpr (is_lp(KIND)) add([&](f32 g, f32 a) -> f32 { return a + pow_abs<(KIND >> 4)>(g, p); });
        else if constexpr (KIND == M_LINF) add([](f32 g, f32 a) -> f32 { return fmaxf(a, g); });
        else if constexpr (KIND == M_L2) add([](f32 g, f32 a) -> f32 { return __fmaf_rd(g, g, a); });
        else add([](f32 g, f32 a) -> f32 { return __fadd_rd(a, g); });
        u32 need = 0;
        b = 0xffffffffu;
#pragma unroll
        for (int q = 0; q < QW; ++q) {
            const f32 v = KIND == M_L2 || KIND == M_L1 ? s[q] * (1.0f - 0x1p-16f) : s[q];
            if (!(v > W.thr[q])) {
                need |= 1u << q;
                b = min(b, __float_as_uint(s[q]));
            }
        }
        return need;
    }
}

// A box in many dimensions is a loose bound: 32 points of a Gaussian in R^32
// spread over +-2 deviations along every axis, so the gaps between two
// clusters nearly vanish one by one. Along the direction from the queries to
// the tile the same points take up a tenth of the distance. For any u,
// |u . (x - q)| <= |u|_p' |x - q|_p (Hoelder, 1/p + 1/p' = 1), so a tile whose
// smallest u . x exceeds u . q by more than |u|_p' times a query's bound holds
// nothing for it. u is the gradient of the distance at the vector D between
// the centres (L2: D; L1: its signs; Lp: sign(D) |D|^(p-1)).
// Rounding: u is what it is, as computed. The projections are sums relative
// to the queries' centre g; each errs by at most (DP + 2) 2^-24 of
// sum |u_k| |x_k - g_k|, which the box corners bound (err: 2^-17 times
// both sides' sums); |u|_p' is taken 2^-9 up.
// The same test between blocks of 128 points, tabulated once (tt_near.cu
// near_separations), replaces the boxes where it is built.
// (100,000 mixture points in R^32: the foreign searches of a spanning tree take
// 45 ms with the boxes alone, 30 with the directions, 9.7 with the table and
// the bounds refreshed; L1.5 lists 13.5 ms, 6.7 with the table.)
template <int DP, int QW>
struct Direction {
    alignas(16) f32 g[DP];     // the queries' centre
    alignas(16) f32 u[DP];
    f32 qy[DP][QW];            // the queries relative to it, coordinate-major
    f32 ext[DP];               // their largest |q_k - g_k|
};
struct NoDirection {};
template <int KIND, int DP>
constexpr bool projects() { return DP >= int(kProjectDim) && KIND != M_LINF; }
template <int KIND, int DP, int QW>
using DirectionOf = typename std::conditional<projects<KIND, DP>(), Direction<DP, QW>, NoDirection>::type;

template <int DP, int QW>
__device__ __forceinline__ void init_direction(const WarpQ<DP, QW>& W, Direction<DP, QW>& D) {
    const u32 lane = threadIdx.x & 31;
    for (u32 k = lane; k < DP; k += 32) {
        f32 lo = W.qt[k][0], hi = lo;
#pragma unroll
        for (int q = 1; q < QW; ++q) lo = fminf(lo, W.qt[k][q]), hi = fmaxf(hi, W.qt[k][q]);
        const f32 g = 0.5f * lo + 0.5f * hi;
        f32 e = 0.0f;
        D.g[k] = g;
#pragma unroll
        for (int q = 0; q < QW; ++q) {
            const f32 y = __fsub_rn(W.qt[k][q], g);
            D.qy[k][q] = y;
            e = fmaxf(e, fabsf(y));
        }
        D.ext[k] = e;
    }
    __syncwarp();
}

__device__ __forceinline__ f32 warp_sum(f32 x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// The queries of `need` that the tile (candidates c, one a lane; `live`: a
// point) may still matter to.
template <int KIND, int DP, int QW>
__device__ __forceinline__ u32 project(const View& v, const WarpQ<DP, QW>& W, Direction<DP, QW>& D, u32 tile,
                                       const f32 (&c)[DP], bool live, u32 need) {
    const u32 lane = threadIdx.x & 31;
    f32 nrm = 0.0f, mag = 0.0f;
#pragma unroll
    for (int h = 0; h < (DP + 31) / 32; ++h) {
        const u32 k = lane + 32 * h;
        if (k < DP) {
            const f32 lo = __ldg(v.abox + (u64(tile) * 2) * DP + k), hi = __ldg(v.abox + (u64(tile) * 2 + 1) * DP + k);
            const f32 g = D.g[k];
            const f32 d = (0.5f * lo + 0.5f * hi) - g;
            f32 u, t;   // the direction, its term of |u|_p'
            if constexpr (KIND == M_L2) {
                u = d;
                t = d * d;
            } else if constexpr (KIND == M_L1) {
                u = d < 0.0f ? -1.0f : 1.0f;
                t = 0.0f;
            } else {
                u = copysignf(pow_abs<0>(d, v.p - 1.0f), d);
                t = pow_abs<0>(u, v.p / (v.p - 1.0f));
            }
            D.u[k] = u;
            nrm += t;
            mag += fabsf(u) * (fmaxf(fabsf(lo - g), fabsf(hi - g)) + D.ext[k]);
        }
    }
    nrm = warp_sum(nrm);
    mag = warp_sum(mag);
    if constexpr (KIND != M_L1)   // terms lost to underflow (each below 2^-126) must not matter
        if (!(nrm >= 0x1p-100f)) return need;
    if constexpr (KIND == M_L2) nrm = sqrtf(nrm);
    else if constexpr (KIND == M_L1) nrm = 1.0f;
    else nrm = pow_abs<0>(nrm, (v.p - 1.0f) / v.p);
    nrm *= 1.0f + 0x1p-9f;
    __syncwarp();
    f32 pc[2] = {0.0f, 0.0f}, pq[2] = {0.0f, 0.0f};
    const u32 ql = lane % QW;
#pragma unroll
    for (int k = 0; k < DP; ++k) {
        const f32 u = D.u[k];
        pc[k & 1] = fmaf(u, __fsub_rn(c[k], D.g[k]), pc[k & 1]);
        pq[k & 1] = fmaf(u, D.qy[k][ql], pq[k & 1]);
    }
    f32 m = pc[0] + pc[1];
    m = live ? m : INFINITY;   // (a NaN candidate: kept below, the difference is NaN or too small)
    const bool odd = __any_sync(0xffffffffu, live && !(m == m));
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const f32 lead = (m - (pq[0] + pq[1])) - 0x1p-16f * mag;
    const bool out = lane < QW && !odd && lead > nrm * W.bnd[lane < QW ? lane : 0] && lead < INFINITY;
    __syncwarp();
    return need & ~__ballot_sync(0xffffffffu, out);
}

// No tile is left out beforehand.
struct SkipNone {
    __device__ __forceinline__ bool tile(u32) const { return false; }
    __device__ __forceinline__ bool super(u32) const { return false; }
    __device__ __forceinline__ void refresh() const {}   // bounds that other warps lower
    static constexpr bool kAlong = false;   // the direction test pays only between blocks that are apart
};

// Walks the tiles in reach of the warp's queries; visit(tile, coordinates,
// candidate id, queries) tests one tile against the queries of a bit mask and
// returns whether a bound may have dropped.
template <int KIND, int DP, int CH, int QW, typename Visit, typename Skip = SkipNone>
__device__ __forceinline__ void walk(const View& v, WarpQ<DP, QW>& W, DirectionOf<KIND, DP, QW>& D, u32 home, Visit&& visit,
                                     Skip skip = Skip{}) {
    const u32 lane = threadIdx.x & 31;
    if constexpr (projects<KIND, DP>()) init_direction<DP, QW>(W, D);
    auto group_thr = [&]() -> f32 {   // the largest bound (-1: none)
        f32 m = -1.0f;
        if constexpr (QW == 1) {
            m = W.thr[0];
        } else {
            if (lane < QW) m = W.thr[lane];
#pragma unroll
            for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        }
        return m;
    };
    // along: worth a test along the direction to the tile
    auto load_visit = [&](u32 tile, u32 need, bool along = true) -> bool {
        f32 c[DP];
        const f32* xt = v.xt + u64(tile) * (DP * kTile) + lane;
#pragma unroll
        for (int k = 0; k < DP; ++k) c[k] = __ldg(xt + k * kTile);
        const u32 cid = __ldg(v.id + tile * kTile + lane);
        if constexpr (projects<KIND, DP>()) {
            if (along && tile != home) {
                need = project<KIND, DP, QW>(v, W, D, tile, c, cid != 0xffffffffu, need);
                if (!need) return false;
            }
        }
        return visit(tile, c, cid, need);
    };
    f32 thr = group_thr();
    if (!skip.tile(home) && load_visit(home, (1u << QW) - 1u)) thr = group_thr();
    const u32 s0 = home / 32;
    // The closest open box of 32 held one a lane (bound bits; ~0: done). The
    // bounds are >= +0, so their bits order like them.
    auto closest = [&](u32 b, u32& src) -> bool {
        const u32 m = __reduce_min_sync(0xffffffffu, b);
        if (m == 0xffffffffu || __uint_as_float(m) * (QW == 1 ? 1.0f : 1.0f - 0x1p-16f) > thr) return false;
        src = u32(__ffs(__ballot_sync(0xffffffffu, b == m)) - 1);
        return true;
    };
    auto descend = [&](u32 s) {
        const u32 t = s * 32 + lane;
        u32 b = 0xffffffffu, need = 0;
        if (t < v.ntiles && t != home && !skip.tile(t))
            need = box_needs<KIND, DP, CH, QW>(v.tbox, v.tpad, t, W, v.p, b);
        u32 src;
        while (closest(b, src)) {
            if (lane == src) b = 0xffffffffu;
            if (load_visit(s * 32 + src, QW == 1 ? 1u : __shfl_sync(0xffffffffu, need, src))) thr = group_thr();
        }
    };
    if constexpr (projects<KIND, DP>()) {
        if (v.sep) {
            // Separations between blocks of points instead of boxes: 32 blocks
            // a test, the closest first, then the block's tiles (each tested
            // along its own direction before its candidates are).
            const u32 hb = home / kBlockTiles;
            const u32 mine = lane < QW ? W.blk[lane] : W.blk[0];
            const bool one = __all_sync(0xffffffffu, mine == hb);
            const u32 br = (v.nblk + 31) / 32, b0 = hb / 32;
            for (u32 r = 0; r < br; ++r) {   // the home round first
                const u32 base = (r == 0 ? b0 : r <= b0 ? r - 1 : r) * 32;
                const u32 t = base + lane;
                u32 b = 0xffffffffu;
                if (t < v.nblk) {
                    f32 d = __ldg(v.sep + u64(hb) * v.nblk + t);
                    if (!one)
                        for (int q = 0; q < QW; ++q) d = fminf(d, __ldg(v.sep + u64(W.blk[q]) * v.nblk + t));
                    b = __float_as_uint(d);
                }
                for (;;) {
                    skip.refresh();
                    f32 far = lane < QW ? W.bnd[lane] : 0.0f;   // the largest distance that still matters
#pragma unroll
                    for (int o = 16; o; o >>= 1) far = fmaxf(far, __shfl_xor_sync(0xffffffffu, far, o));
                    const u32 m = __reduce_min_sync(0xffffffffu, b);
                    if (m == 0xffffffffu || __uint_as_float(m) > far) break;
                    const u32 src = u32(__ffs(__ballot_sync(0xffffffffu, b == m)) - 1);
                    if (lane == src) b = 0xffffffffu;
                    for (u32 tile = (base + src) * kBlockTiles;
                         tile < min(v.ntiles, (base + src + 1) * kBlockTiles); ++tile)
                        if (tile != home && !skip.tile(tile)) load_visit(tile, (1u << QW) - 1u, Skip::kAlong || m != 0u);
                }
            }
            return;
        }
    }
    if (!skip.super(s0)) descend(s0);
    const u32 rounds = (v.nsup + 31) / 32, r0 = s0 / 32;
    for (u32 r = 0; r < rounds; ++r) {   // the home round first
        const u32 base = (r == 0 ? r0 : r <= r0 ? r - 1 : r) * 32;
        const u32 s = base + lane;
        u32 b = 0xffffffffu;
        if (s < v.nsup && s != s0 && !skip.super(s))
            box_needs<KIND, DP, CH, QW>(v.sbox, v.spad, s, W, v.p, b);
        u32 src;
        while (closest(b, src)) {
            if (lane == src) b = 0xffffffffu;
            descend(base + src);
        }
    }
}

// Queries p0 .. p0 + QW - 1 of the order into W; thr0 is every query's first
// bound. Returns the mask of lanes (< QW) that hold a query.
template <int DP, int QW>
__device__ __forceinline__ void load_queries(const View& v, u32 p0, f32 thr0, WarpQ<DP, QW>& W) {
    const u32 lane = threadIdx.x & 31;
    for (u32 e = lane; e < QW * DP; e += 32) {
        const u32 q = e / DP, k = e % DP, p = p0 + q;
        W.q[q][k] = W.qt[k][q] = p < v.n ? v.xt[u64(p / kTile) * (DP * kTile) + k * kTile + p % kTile] : 0.0f;
    }
    if (lane < QW) {
        const u32 p = p0 + lane;
        W.thr[lane] = p < v.n ? thr0 : -1.0f;
        W.bnd[lane] = p < v.n ? INFINITY : 0.0f;
        W.blk[lane] = p0 / (kTile * kBlockTiles);
        W.own[lane] = p < v.n ? v.id[p] : 0xffffffffu;
    }
    __syncwarp();
}

template <int DP>
struct RegDiff {
    const f32* q;
    const f32 (&c)[DP];
    __device__ __forceinline__ f32 operator()(int k) const { return __fsub_rn(q[k], c[k]); }
};

// ---- k nearest neighbours ---------------------------------------------------
// Each query's list is 32 sorted keys (distance bits << 32 | id), one a lane;
// the first k are the answer. Distances are >= +0, so key order is the
// (distance, id) order of the lists; empty slots hold (+inf, ~0), and a NaN
// distance orders above them and never enters.
constexpr u64 kEmpty = 0x7f800000ffffffffull;

__device__ __forceinline__ u64 shfl64(u64 x, u32 src) { return __shfl_sync(0xffffffffu, x, src); }

// Up to 32 keys (lanes of `mask`) into the sorted list L; kth = its k-th key.
__device__ __forceinline__ void merge_keys(u64& L, u64& kth, u32 k, u64 key, u32 mask) {
    const u32 lane = threadIdx.x & 31;
    if (__popc(mask) <= 12) {   // one by one: about 16 instructions a key
        while (mask) {
            const u64 kk = shfl64(key, u32(__ffs(mask) - 1));
            mask &= mask - 1;
            if (kk >= kth) continue;
            const u32 pos = __popc(__ballot_sync(0xffffffffu, L < kk));
            const u64 up = __shfl_up_sync(0xffffffffu, L, 1);
            L = lane < pos ? L : lane == pos ? kk : up;
            kth = shfl64(L, k - 1);
        }
    } else {   // sort them, then the 32 smallest of the two sorted halves: about 200 in all
        u64 x = (mask >> lane) & 1u ? key : ~0ull;
#pragma unroll
        for (u32 size = 2; size <= 32; size <<= 1) {
#pragma unroll
            for (u32 stride = size >> 1; stride; stride >>= 1) {
                const u64 y = __shfl_xor_sync(0xffffffffu, x, stride);
                const bool up = ((lane & size) == 0) == ((lane & stride) == 0);
                x = up ? (x < y ? x : y) : (x < y ? y : x);
            }
        }
        const u64 r = shfl64(x, 31 - lane);
        L = L < r ? L : r;   // bitonic
#pragma unroll
        for (u32 stride = 16; stride; stride >>= 1) {
            const u64 y = __shfl_xor_sync(0xffffffffu, L, stride);
            L = (lane & stride) == 0 ? (L < y ? L : y) : (L < y ? y : L);
        }
        kth = shfl64(L, k - 1);
    }
}

// 100,000 uniform points in R^3, k = 15, L2: 0.225 ms (exhaustive scan 31.55
// ms); 20,011 x 8 Gaussian points, Linf, k = 10: 0.36 ms (2.9 ms). Latency
// bound: the walk's loads and shuffles follow each other.
template <int KIND, int DP, int CH, int QW>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_knn(View v, u32 k, u32* __restrict__ ids, f32* __restrict__ dists) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, QW> sw[kWarps];
    __shared__ DirectionOf<KIND, DP, QW> sd[projects<KIND, DP>() ? kWarps : 1];
    __shared__ u64 slist[kWarps][QW][32];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 p0 = (blockIdx.x * kWarps + w) * QW;
    if (p0 >= v.n) return;
    WarpQ<DP, QW>& W = sw[w];
    load_queries<DP, QW>(v, p0, INFINITY, W);
    u64(&list)[QW][32] = slist[w];
#pragma unroll
    for (int q = 0; q < QW; ++q) list[q][lane] = kEmpty;
    __syncwarp();
    walk<KIND, DP, CH, QW>(v, W, sd[projects<KIND, DP>() ? w : 0], p0 / kTile, [&](u32, const f32(&c)[DP], u32 cid, u32 need) -> bool {
        bool dropped = false;
#pragma unroll 1
        for (; need; need &= need - 1) {
            const u32 q = QW == 1 ? 0u : u32(__ffs(need) - 1);
            const f32 s = eval<KIND, DP, CH>(RegDiff<DP>{W.q[q], c});
            const f32 tq = W.thr[q];
            // (past the points: id ~0; past the queries: bound -1)
            const bool pass = cid != W.own[q] && cid != 0xffffffffu && !(s > tq);
            if (!__any_sync(0xffffffffu, pass)) continue;
            const f32 d = KIND == M_L2 ? __fsqrt_rn(s) : s;
            const u64 key = (u64(__float_as_uint(d)) << 32) | cid;
            u64 L = list[q][lane];
            u64 kth = shfl64(L, k - 1);
            const u32 mask = __ballot_sync(0xffffffffu, pass && key < kth);
            if (!mask) continue;
            merge_keys(L, kth, k, key, mask);
            list[q][lane] = L;
            if (lane == 0) {
                const f32 dk = __uint_as_float(u32(kth >> 32));
                W.thr[q] = bound_of<KIND>(dk);
                if constexpr (projects<KIND, DP>()) W.bnd[q] = bound_margin(dk);
            }
            __syncwarp();
            dropped = true;
        }
        return dropped;
    });
#pragma unroll 1
    for (u32 q = 0; q < QW; ++q) {
        if (p0 + q >= v.n) break;
        const u64 L = list[q][lane];
        const u64 o = u64(W.own[q]) * k + lane;
        if (lane < k) {
            ids[o] = u32(L);
            if (dists) dists[o] = __uint_as_float(u32(L >> 32));
        }
    }
}

// Lp lists. A candidate of a query with k-th distance B is evaluated exactly
// when its power sum F = sum |d_k|^p (fast) is at most
//   T = B^p (fast) (1 + (p + 1) 2^-12).
// The reference's distance (lp_parts, lp_root) is M powf(s, 1/p) with s the
// sum of its power series of |d_k| / M: the series' log2 (arguments above
// 1e-30) errs by less than 2^-16, so a term by a factor within
// 1 +- (p 2^-16 + 2^-18), the terms it clamps by less than 2^-126 of a sum
// that is at least about 1, and the root by p 2^-22 of the power. F and T err by
// p 2^-15 each (lg2.approx within 2^-22 of a logarithm below 128, ex2.approx
// 2^-22, sums of 64 terms 2^-18). Together below p 2^-13.6 + 2^-16 for p <= kLpMax, a
// third of the margin. T outside [2^-100, 2^100], where powers
// under- or overflow, filters nothing. The gap vector of a box goes through the same sum: the power sums of the
// coordinate differences, as rounded, are at least the gap's.
// Survivors are queued and evaluated 32 at a time, one a lane, so that the
// long exact path runs in full warps.
// 100,000 x 32 mixture points, L1.5, k = 15: 6.7 ms (exhaustive scan with early
// exits: 390 ms). Bound by issue and the
// special-function unit (one square root a coordinate).
template <int KIND>
__device__ __forceinline__ f32 lp_thr(f32 d, f32 p) {
    if (!(d < INFINITY)) return INFINITY;
    const f32 t = pow_abs<(KIND >> 4)>(d, p) * (1.0f + (p + 1.0f) * 0x1p-12f);
    return t >= 0x1p-100f && t <= 0x1p100f ? t : INFINITY;
}

struct TileCol {   // coordinate k of one candidate
    const f32* x;
    __device__ __forceinline__ f32 operator()(u32 k) const { return __ldg(x + k * kTile); }
};

template <int KIND, int DP, int QW>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_knn_lp(View v, u32 dim, u32 k, u32* __restrict__ ids, f32* __restrict__ dists) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, QW> sw[kWarps];
    __shared__ DirectionOf<KIND, DP, QW> sd[projects<KIND, DP>() ? kWarps : 1];
    __shared__ u64 slist[kWarps][QW][32];
    __shared__ u32 spos[kWarps][64];   // survivors: position in the order, query (a ring)
    __shared__ u8 sq[kWarps][64];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const u32 p0 = (blockIdx.x * kWarps + w) * QW;
    if (p0 >= v.n) return;
    WarpQ<DP, QW>& W = sw[w];
    load_queries<DP, QW>(v, p0, INFINITY, W);
    u64(&list)[QW][32] = slist[w];
#pragma unroll
    for (int q = 0; q < QW; ++q) list[q][lane] = kEmpty;
    __syncwarp();
    u32 head = 0, count = 0;
    // evaluates the first `cnt` (at most 32) survivors
    auto flush = [&](u32 cnt) {
        __syncwarp();
        const bool in = lane < cnt;
        const u32 pos = in ? spos[w][(head + lane) & 63] : 0, q = in ? sq[w][(head + lane) & 63] : 0;
        u64 key = ~0ull;
        if (in) {
            f32 M, sum;
            lp_parts(Row{W.q[q]}, TileCol{v.xt + u64(pos / kTile) * (DP * kTile) + pos % kTile}, dim, v.p, M, sum);
            const f32 bd = __uint_as_float(u32(list[q][k - 1] >> 32));
            if (!(lp_root_lower(M, sum, v.p) > bd))
                key = (u64(__float_as_uint(lp_root(M, sum, v.p))) << 32) | v.id[pos];
        }
        for (u32 open = __ballot_sync(0xffffffffu, key != ~0ull); open;) {
            const u32 qq = __shfl_sync(0xffffffffu, q, __ffs(open) - 1);
            const u32 all = __ballot_sync(0xffffffffu, q == qq) & open;
            open &= ~all;
            u64 L = list[qq][lane];
            u64 kth = shfl64(L, k - 1);
            const u32 mask = __ballot_sync(0xffffffffu, key < kth) & all;
            if (!mask) continue;
            merge_keys(L, kth, k, key, mask);
            list[qq][lane] = L;
            if (lane == 0) {
                const f32 dk = __uint_as_float(u32(kth >> 32));
                W.thr[qq] = lp_thr<KIND>(dk, v.p);
                if constexpr (projects<KIND, DP>()) W.bnd[qq] = bound_margin(dk);
            }
            __syncwarp();
        }
        head += cnt;
        count -= cnt;
        __syncwarp();
    };
    walk<KIND, DP, 0, QW>(v, W, sd[projects<KIND, DP>() ? w : 0], p0 / kTile, [&](u32 tile, const f32(&c)[DP], u32 cid, u32 need) -> bool {
        bool dropped = false;
#pragma unroll 1
        for (; need; need &= need - 1) {
            const u32 q = QW == 1 ? 0u : u32(__ffs(need) - 1);
            const f32 s = eval<KIND, DP, 0>(RegDiff<DP>{W.q[q], c}, v.p);
            const bool pass = cid != W.own[q] && cid != 0xffffffffu && !(s > W.thr[q]);
            const u32 m = __ballot_sync(0xffffffffu, pass);
            if (!m) continue;
            if (pass) {
                const u32 o = (head + count + __popc(m & lt)) & 63;
                spos[w][o] = tile * kTile + lane;
                sq[w][o] = u8(q);
            }
            count += __popc(m);
            if (count >= 32) {
                flush(32);
                dropped = true;
            }
        }
        return dropped;
    });
    if (count) flush(count);
#pragma unroll 1
    for (u32 q = 0; q < QW; ++q) {
        if (p0 + q >= v.n) break;
        const u64 L = list[q][lane];
        const u64 o = u64(W.own[q]) * k + lane;
        if (lane < k) {
            ids[o] = u32(L);
            if (dists) dists[o] = __uint_as_float(u32(L >> 32));
        }
    }
}

// ---- nearest point of another component -------------------------------------
// One Borůvka round's proposals (tt_mst.cu): for every listed query (positions
// in the order, `qlist`, ~0 entries skipped) its minimum (distance, id) over
// the points of other components, near[id] = distance bits << 32 | id. A
// tile, or a super tile, whose points all share the queries' component is left
// out (tcomp, scomp: the shared component, or kMixed).
// Only a component's best proposal counts, so a query starts from the bound
// bd[component], the best its component has so far (distance bits), takes up
// what other warps find meanwhile and publishes its own: candidates above the
// bound cannot be the component's minimum, those at the bound still compete by
// edge index. A query without a candidate within the bound leaves ~0.
constexpr u32 kMixed = 0xfffffffeu, kNoComp = 0xffffffffu;

template <int KIND, typename WQ>
struct SkipComp {
    const u32* tcomp;
    const u32* scomp;
    u32 comp;   // the queries' shared component, or kNoComp
    WQ* W;
    const u32* cq;   // the queries' components
    static constexpr bool kAlong = true;   // a block may hold points of two clusters
    u32 queries;
    const u32* bd;
    // takes up the components' bounds as other warps have left them
    __device__ __forceinline__ void refresh() const {
        const u32 lane = threadIdx.x & 31;
        if (lane < queries && cq[lane] != kNoComp) {
            const u32 b = *reinterpret_cast<const volatile u32*>(bd + cq[lane]);
            if (b != 0xffffffffu) {
                W->thr[lane] = fminf(W->thr[lane], bound_of<KIND>(__uint_as_float(b)));
                W->bnd[lane] = fminf(W->bnd[lane], bound_margin(__uint_as_float(b)));
            }
        }
        __syncwarp();
    }
    __device__ __forceinline__ bool tile(u32 t) const { return __ldg(tcomp + t) == comp; }
    __device__ __forceinline__ bool super(u32 s) const { return __ldg(scomp + s) == comp; }
};

template <int KIND, int DP, int CH, int QW>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_foreign(View v, const u32* __restrict__ cpos, const u32* __restrict__ tcomp, const u32* __restrict__ scomp,
                   const u32* __restrict__ qlist, const u32* __restrict__ nq, u32* bd,
                   unsigned long long* __restrict__ near) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, QW> sw[kWarps];
    __shared__ DirectionOf<KIND, DP, QW> sd[projects<KIND, DP>() ? kWarps : 1];
    __shared__ u64 sbest[kWarps][QW];
    __shared__ u32 scq[kWarps][QW];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 g0 = (blockIdx.x * kWarps + w) * QW;
    if (g0 >= *nq) return;
    WarpQ<DP, QW>& W = sw[w];
    u64(&best)[QW] = sbest[w];
    u32(&cq)[QW] = scq[w];
    u32 mypos = 0xffffffffu, mycomp = kNoComp;
    if (lane < QW) {
        mypos = qlist[g0 + lane];   // (the list is padded to whole groups)
        const bool in = mypos != 0xffffffffu;
        mycomp = in ? cpos[mypos] : kNoComp;
        const u32 b = in ? *reinterpret_cast<volatile u32*>(bd + mycomp) : 0u;
        cq[lane] = mycomp;
        best[lane] = in ? (u64(b) << 32) | 0xffffffffu : 0ull;
        W.own[lane] = in ? v.id[mypos] : 0xffffffffu;
        W.thr[lane] = !in ? -1.0f : b == 0xffffffffu ? INFINITY : bound_of<KIND>(__uint_as_float(b));
        W.bnd[lane] = !in ? 0.0f : b == 0xffffffffu ? INFINITY : bound_margin(__uint_as_float(b));
    }
    __syncwarp();
    const u32 first = __ballot_sync(0xffffffffu, mypos != 0xffffffffu);   // never empty: lists start groups with a query
    const u32 p_home = __shfl_sync(0xffffffffu, mypos, __ffs(first) - 1);
    const u32 c_home = __shfl_sync(0xffffffffu, mycomp, __ffs(first) - 1);
    if (lane < QW) W.blk[lane] = (mypos != 0xffffffffu ? mypos : p_home) / (kTile * kBlockTiles);
    const bool one = __all_sync(0xffffffffu, mypos == 0xffffffffu || mycomp == c_home);
#pragma unroll 1
    for (u32 e = lane; e < QW * DP; e += 32) {
        const u32 q = e / DP, k = e % DP;
        const u32 p = W.own[q] != 0xffffffffu ? qlist[g0 + q] : p_home;   // (a missing query repeats the first)
        W.q[q][k] = W.qt[k][q] = v.xt[u64(p / kTile) * (DP * kTile) + k * kTile + p % kTile];
    }
    __syncwarp();
    const SkipComp<KIND, WarpQ<DP, QW>> skip{tcomp, scomp, one ? c_home : kNoComp, &W, cq, QW, bd};
    walk<KIND, DP, CH, QW>(
        v, W, sd[projects<KIND, DP>() ? w : 0], p_home / kTile,
        [&](u32 tile, const f32(&c)[DP], u32 cid, u32 need) -> bool {
            const u32 cc = __ldg(cpos + tile * kTile + lane);   // kNoComp past the points
            bool dropped = false;
#pragma unroll 1
            for (; need; need &= need - 1) {
                const u32 q = QW == 1 ? 0u : u32(__ffs(need) - 1);
                const f32 s = eval<KIND, DP, CH>(RegDiff<DP>{W.q[q], c});
                const bool pass = cid != 0xffffffffu && cc != cq[q] && !(s > W.thr[q]);
                if (!__any_sync(0xffffffffu, pass)) continue;
                const f32 d = KIND == M_L2 ? __fsqrt_rn(s) : s;
                const u64 old = best[q];
                const u64 key = (u64(__float_as_uint(d)) << 32) | cid;
                const bool take = pass && key < old;
                const u32 dm = __reduce_min_sync(0xffffffffu, take ? u32(key >> 32) : 0xffffffffu);
                const u32 im = __reduce_min_sync(0xffffffffu, take && u32(key >> 32) == dm ? cid : 0xffffffffu);
                if (im == 0xffffffffu) continue;
                if (lane == 0) {
                    best[q] = (u64(dm) << 32) | im;
                    // the component's bound: ours, or a smaller one found meanwhile
                    const u32 seen = atomicMin(bd + cq[q], dm);
                    W.thr[q] = bound_of<KIND>(__uint_as_float(min(seen, dm)));
                    W.bnd[q] = bound_margin(__uint_as_float(min(seen, dm)));
                }
                __syncwarp();
                dropped = true;
            }
            return dropped;
        },
        skip);
    if (lane < QW && mypos != 0xffffffffu) {
        const u64 k = best[lane];
        near[W.own[lane]] = u32(k) == 0xffffffffu ? ~0ull : k;
    }
}

// ---- radius graph -----------------------------------------------------------
// Row lengths (cnt by original id) and the longest row, then the rows: a warp
// collects a row's ids and distances in shared memory, orders them by id and
// writes the row. The order is a bitonic sort of 32-bit keys in registers: an
// id relative to the row's smallest, above the entry's place in shared memory,
// 1 to 32 keys a lane by the row's length. Ids that spread over more than
// 2^22 are sorted in shared memory.
// 50,000 uniform points in R^3, 240 neighbours: count 0.14 ms, fill 0.48 ms
// with 64-bit keys sorted in shared memory, now 0.20 (exhaustive scans 4.2 and
// 4.05 ms). Two row capacities (launch by the longest row): the shared memory
// of the larger leaves 24 warps an SM.
constexpr u32 kRowBits = 10;   // of an entry's place
static_assert(kRadiusRow <= 1u << kRowBits, "an entry's place fits its bits");

// A row's entries in shared memory; the ids' words take the sorted keys (a
// padding word after every 32, so that a lane's K stores meet no other's bank).
template <u32 ROW>
struct Row {
    u32 id[ROW + ROW / 32];
    f32 d[ROW];
};

template <int K, u32 ROW>
__device__ __forceinline__ void sort_row(Row<ROW>& R, u32 len, u32 least, u32* __restrict__ ci, f32* __restrict__ wt) {
    const u32 lane = threadIdx.x & 31;
    u32 key[K];
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const u32 e = i * 32 + lane;
        key[i] = e < len ? (R.id[e] - least) << kRowBits | e : 0xffffffffu;
    }
    sort_lane_keys<K>(key);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const u32 o = lane * K + i;
        R.id[o + o / 32] = key[i];
    }
    __syncwarp();
    for (u32 e = lane; e < len; e += 32) {
        const u32 k = R.id[e + e / 32];
        ci[e] = (k >> kRowBits) + least;
        wt[e] = R.d[k & ((1u << kRowBits) - 1u)];
    }
}

// ROW: the row capacity (0: count only).
template <int KIND, int DP, int CH, u32 ROW>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_radius(View v, f32 tau, f32 bound, u64* __restrict__ cnt, u32* __restrict__ longest,
                  const u64* __restrict__ rp, u32* __restrict__ ci, f32* __restrict__ wt) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, 1> sw[kWarps];
    __shared__ DirectionOf<KIND, DP, 1> sd[projects<KIND, DP>() ? kWarps : 1];
    __shared__ Row<ROW ? ROW : 32> srow[ROW ? kWarps : 1];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 p0 = blockIdx.x * kWarps + w;
    if (p0 >= v.n) return;
    WarpQ<DP, 1>& W = sw[w];
    load_queries<DP, 1>(v, p0, bound, W);
    auto& R = srow[ROW ? w : 0];
    u32 len = 0, least = 0xffffffffu, most = 0;
    walk<KIND, DP, CH, 1>(v, W, sd[projects<KIND, DP>() ? w : 0], p0 / kTile, [&](u32, const f32(&c)[DP], u32 cid, u32) -> bool {
        const f32 s = eval<KIND, DP, CH>(RegDiff<DP>{W.q[0], c});
        bool pass = cid != W.own[0] && cid != 0xffffffffu && s <= bound;
        if (!__any_sync(0xffffffffu, pass)) return false;
        const f32 d = KIND == M_L2 ? __fsqrt_rn(s) : s;
        pass = pass && d <= tau;
        const u32 m = __ballot_sync(0xffffffffu, pass);
        if constexpr (ROW > 0) {
            const u32 o = len + __popc(m & ((1u << lane) - 1u));
            if (pass && o < ROW) {
                R.id[o] = cid;
                R.d[o] = d;
                least = min(least, cid);
                most = max(most, cid);
            }
        }
        len += __popc(m);
        return false;
    });
    const u32 own = W.own[0];
    if constexpr (ROW == 0) {
        if (lane == 0) {
            cnt[own] = len;
            if (len > kRadiusRow / 2) atomicMax(longest, len);
        }
    } else {
        const u64 b = rp[own];
        const u32 m = min(len, ROW);
        if (m == 0) return;
        least = __reduce_min_sync(0xffffffffu, least);
        most = __reduce_max_sync(0xffffffffu, most);
        __syncwarp();
        if (most - least < (1u << (32 - kRowBits)) - 1u) {   // (the largest key is the padding's)
            if (m <= 32) sort_row<1, ROW>(R, m, least, ci + b, wt + b);
            else if (m <= 128) sort_row<4, ROW>(R, m, least, ci + b, wt + b);
            else if (m <= 256) sort_row<8, ROW>(R, m, least, ci + b, wt + b);
            else if (ROW <= 512 || m <= 512) sort_row<16, ROW>(R, m, least, ci + b, wt + b);
            else sort_row<ROW / 32, ROW>(R, m, least, ci + b, wt + b);
            return;
        }
        u32 P = 32;
        while (P < m) P <<= 1;
        for (u32 i = m + lane; i < P; i += 32) R.id[i] = 0xffffffffu;
        __syncwarp();
        for (u32 size = 2; size <= P; size <<= 1) {
            for (u32 stride = size >> 1; stride; stride >>= 1) {
                for (u32 i = lane; i < P / 2; i += 32) {
                    const u32 lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                    const u32 x = R.id[lo], y = R.id[hi];
                    if ((x > y) == ((lo & size) == 0)) {
                        const f32 t = R.d[lo];
                        R.id[lo] = y;
                        R.id[hi] = x;
                        R.d[lo] = R.d[hi];
                        R.d[hi] = t;
                    }
                }
                __syncwarp();
            }
        }
        for (u32 i = lane; i < m; i += 32) {
            ci[b + i] = R.id[i];
            wt[b + i] = R.d[i];
        }
    }
}

template <int KIND, int DP, int CH>
void launch_knn(tt_ctx* c, const View& v, u32 k, u32* ids, f32* dists) {
    constexpr int QW = queries_per_warp(DP);
    auto go = [&](auto qw) {
        constexpr int Q = decltype(qw)::value;
        launch_pdl(k_near_knn<KIND, DP, CH, Q>, div_up(div_up(v.n, Q), kWarps), 32 * kWarps, 0, c->stream, v, k, ids, dists);
    };
    // few points: more warps count for more than the reuse of a tile's loads
    // (3,000 x 24 uniform points 0.35 ms with 8 queries a warp, 0.25 with 4;
    // 16,000 x 16 mixture points 0.76 and 0.85)
    if (DP >= 16 && v.n <= kFewPoints) go(std::integral_constant<int, QW >= 4 ? QW / 2 : QW>{});
    else go(std::integral_constant<int, QW>{});
    TT_LAUNCH("k_near_knn");
    ++c->launches;
}

// f(padded dimension, chunks) for dim, as compile-time constants
template <int KIND, typename F>
void with_dim(u32 dim, F&& f) {
    using std::integral_constant;
    auto go = [&](auto dp, auto ch) {
        // (a max, and Lp's filter: no lane order)
        if constexpr (KIND == M_LINF || is_lp(KIND)) f(dp, integral_constant<int, 0>{});
        else f(dp, ch);
    };
#define TT_D(DP, CH) go(integral_constant<int, DP>{}, integral_constant<int, CH>{})
    if (dim <= 2) TT_D(2, 0);
    else if (dim == 3) TT_D(3, 0);
    else if (dim == 4) TT_D(4, 0);
    else if (dim <= 8) TT_D(8, 0);
    else if (dim <= 15) TT_D(16, 0);
    else if (dim == 16) TT_D(16, 1);
    else if (dim <= 31) TT_D(32, 1);
    else if (dim == 32) TT_D(32, 2);
    else if (dim <= 47) TT_D(48, 2);
    else if (dim == 48) TT_D(48, 3);
    else if (dim <= 63) TT_D(64, 3);
    else TT_D(64, 4);
#undef TT_D
}

template <int KIND>
void near_knn(tt_ctx* c, const View& v, u32 dim, u32 k, u32* ids, f32* dists) {
    with_dim<KIND>(dim, [&](auto dp, auto ch) {
        launch_knn<KIND, decltype(dp)::value, decltype(ch)::value>(c, v, k, ids, dists);
    });
}

template <int KIND>
void near_foreign(tt_ctx* c, const View& v, u32 dim, const u32* cpos, const u32* tcomp, const u32* scomp,
                  const u32* qlist, const u32* nq, u32* bd, unsigned long long* near) {
    with_dim<KIND>(dim, [&](auto dp, auto ch) {
        constexpr int QW = queries_per_warp(decltype(dp)::value);
        launch_pdl(k_near_foreign<KIND, decltype(dp)::value, decltype(ch)::value, QW>,
                   div_up(u64(v.ntiles) * kTile, QW * kWarps), 32 * kWarps, 0, c->stream, v, cpos, tcomp, scomp, qlist,
                   nq, bd, near);
        TT_LAUNCH("k_near_foreign");
        ++c->launches;
    });
}

template <int KIND, u32 ROW>
void radius_pass(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest, const u64* rp, u32* ci, f32* w) {
    // the largest eval value a kept pair can have (host copy of bound_of)
    f32 bound = tau;
    if (KIND == M_L2 && tau < INFINITY) {
        const double up = double(std::nextafter(tau, INFINITY));
        bound = std::nextafter(f32(up * up), INFINITY);
    }
    with_dim<KIND>(dim, [&](auto dp, auto ch) {
        if constexpr (decltype(dp)::value <= 8) {
            launch_pdl(k_near_radius<KIND, decltype(dp)::value, decltype(ch)::value, ROW>, div_up(v.n, kWarps),
                       32 * kWarps, 0, c->stream, v, tau, bound, cnt, longest, rp, ci, w);
            TT_LAUNCH("k_near_radius");
            ++c->launches;
        }
    });
}

template <int KIND>
void near_radius_count(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest) {
    radius_pass<KIND, 0>(c, v, dim, tau, cnt, longest, nullptr, nullptr, nullptr);
}
template <int KIND>
void near_radius_fill(tt_ctx* c, const View& v, u32 dim, f32 tau, u32 longest, const u64* rp, u32* ci, f32* w) {
    if (longest <= kRadiusRow / 2) radius_pass<KIND, kRadiusRow / 2>(c, v, dim, tau, nullptr, nullptr, rp, ci, w);
    else radius_pass<KIND, kRadiusRow>(c, v, dim, tau, nullptr, nullptr, rp, ci, w);
}

// Lp lists of one power class (a translation unit each)
template <int CLS>
void knn_lp_class(tt_ctx* c, const View& v, u32 dim, u32 k, u32* ids, f32* dists) {
    constexpr int KIND = M_LP + 16 * CLS;
    with_dim<KIND>(dim, [&](auto dp, auto) {
        constexpr int DP = decltype(dp)::value, QW = queries_per_warp(DP);
        auto go = [&](auto qw) {
            constexpr int Q = decltype(qw)::value;
            launch_pdl(k_near_knn_lp<KIND, DP, Q>, div_up(div_up(v.n, Q), kWarps), 32 * kWarps, 0, c->stream, v, dim, k,
                       ids, dists);
        };
        if (DP >= 16 && v.n <= kFewPoints) go(std::integral_constant<int, QW >= 4 ? QW / 2 : QW>{});   // (as launch_knn)
        else go(std::integral_constant<int, QW>{});
        TT_LAUNCH("k_near_knn_lp");
        ++c->launches;
    });
}

#endif  // TT_NEAR_IMPL

}  // namespace near
}  // namespace tt
