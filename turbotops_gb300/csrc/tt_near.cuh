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
// registers and tested against the QW queries in turn (their coordinates
// broadcast from shared memory), so more queries a warp reuse the tile's
// loads at the price of a larger common box: 1 up to four dimensions, 8 from
// 32 on.
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
// (Non-integer and integer Lp have no such evaluation: they stay with the
// exhaustive scan.) Coordinates padded with zeros beyond the dimension add
// exact zeros to the sums, in the same lane order.
#pragma once
#include "tt_internal.cuh"
#include "tt_metric.cuh"

namespace tt {
namespace near {

constexpr u32 kTile = 32;
constexpr u32 kWarps = 4;          // warps a block
constexpr u32 kMaxDim = 64;

// The points in order. Boxes: lower corners, then upper ones, coordinate by
// coordinate (row k: the tiles' values, padded to `tpad` / `spad` columns).
struct View {
    const f32* xt = nullptr;   // [ntiles][dp][32]
    const u32* id = nullptr;   // [ntiles * 32]: original ids, ~0 past n
    const f32* tbox = nullptr;   // [2 * dp][tpad]
    const f32* sbox = nullptr;   // [2 * dp][spad]
    u32 n = 0, ntiles = 0, nsup = 0, tpad = 0, spad = 0;
};

// Coordinates held for `dim` (zero-padded) and 16-coordinate chunks in the
// metric's lane order (l2_sq_acc, l1_acc: dim / 16; linf is order-free).
inline u32 padded_dim(u32 dim) {
    return dim <= 4 ? (dim < 2 ? 2 : dim) : dim <= 8 ? 8 : dim <= 16 ? 16 : dim <= 32 ? 32 : dim <= 48 ? 48 : 64;
}

// Queries a warp takes at once (tt_near.cuh's header).
constexpr u32 queries_per_warp(u32 dp) { return dp <= 4 ? 1 : dp <= 8 ? 2 : dp <= 16 ? 4 : 8; }

// tt_near.cu
View near_order(tt_ctx* c, const f32* x, u32 n, u32 dim);

// tt_near_<kind>.cu
template <int KIND>
void near_knn(tt_ctx* c, const View& v, u32 dim, u32 k, u32* ids, f32* dists);
template <int KIND>
void near_radius_count(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest);
template <int KIND>
void near_radius_fill(tt_ctx* c, const View& v, u32 dim, f32 tau, const u64* rp, u32* ci, f32* w);
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

// The metric's evaluation before its final root (L2: the squared sum), of
// d[k] = q[k] - c[k], the query's coordinates in shared memory, the
// candidate's (or the gap's) in registers; the lane order of tt_metric.cuh
// for dim coordinates with CH = dim / 16 chunks, zero-padded to DP.
template <int KIND, int DP, int CH, typename Diff>
__device__ __forceinline__ f32 eval(const Diff& diff) {
    if constexpr (KIND == M_LINF) {
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

template <int DP>
constexpr int row_floats() { return (DP + 3) / 4 * 4; }

// One warp's queries: coordinates, common box, bounds.
template <int DP, int QW>
struct WarpQ {
    alignas(16) f32 q[QW][row_floats<DP>()];
    f32 lo[DP], hi[DP];
    f32 thr[QW];   // eval values above it cannot matter (negative: no query)
    u32 own[QW];
};

// Lower bound of box column t against the warp's box.
template <int KIND, int DP, int CH, int QW>
__device__ __forceinline__ f32 box_bound(const f32* __restrict__ box, u32 pad, u32 t, const WarpQ<DP, QW>& W) {
    return eval<KIND, DP, CH>([&](int k) -> f32 {
        const f32 lo = __ldg(box + u64(k) * pad + t), hi = __ldg(box + u64(DP + k) * pad + t);
        // (infinities that cancel leave a NaN, which fmaxf drops: a gap of 0)
        return fmaxf(fmaxf(__fsub_rn(lo, W.hi[k]), __fsub_rn(W.lo[k], hi)), 0.0f);
    });
}

// No tile is left out beforehand.
struct SkipNone {
    __device__ __forceinline__ bool tile(u32) const { return false; }
    __device__ __forceinline__ bool super(u32) const { return false; }
};

// Walks the tiles in reach of the warp's queries; visit(tile, coordinates,
// candidate id) tests one tile and returns whether a bound may have dropped.
template <int KIND, int DP, int CH, int QW, typename Visit, typename Skip = SkipNone>
__device__ __forceinline__ void walk(const View& v, WarpQ<DP, QW>& W, u32 home, Visit&& visit, Skip skip = Skip{}) {
    const u32 lane = threadIdx.x & 31;
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
    auto load_visit = [&](u32 tile) -> bool {
        f32 c[DP];
        const f32* xt = v.xt + u64(tile) * (DP * kTile) + lane;
#pragma unroll
        for (int k = 0; k < DP; ++k) c[k] = __ldg(xt + k * kTile);
        return visit(tile, c, __ldg(v.id + tile * kTile + lane));
    };
    f32 thr = group_thr();
    if (!skip.tile(home) && load_visit(home)) thr = group_thr();
    const u32 s0 = home / 32;
    // The closest open box of 32 held one a lane (bound bits; ~0: done). The
    // bounds are >= +0, so their bits order like them.
    auto closest = [&](u32 b, u32& src) -> bool {
        const u32 m = __reduce_min_sync(0xffffffffu, b);
        if (m == 0xffffffffu || __uint_as_float(m) > thr) return false;
        src = u32(__ffs(__ballot_sync(0xffffffffu, b == m)) - 1);
        return true;
    };
    auto descend = [&](u32 s) {
        const u32 t = s * 32 + lane;
        u32 b = 0xffffffffu;
        if (t < v.ntiles && t != home && !skip.tile(t))
            b = __float_as_uint(box_bound<KIND, DP, CH, QW>(v.tbox, v.tpad, t, W));
        u32 src;
        while (closest(b, src)) {
            if (lane == src) b = 0xffffffffu;
            if (load_visit(s * 32 + src)) thr = group_thr();
        }
    };
    if (!skip.super(s0)) descend(s0);
    const u32 rounds = (v.nsup + 31) / 32, r0 = s0 / 32;
    for (u32 r = 0; r < rounds; ++r) {   // the home round first
        const u32 base = (r == 0 ? r0 : r <= r0 ? r - 1 : r) * 32;
        const u32 s = base + lane;
        u32 b = 0xffffffffu;
        if (s < v.nsup && s != s0 && !skip.super(s))
            b = __float_as_uint(box_bound<KIND, DP, CH, QW>(v.sbox, v.spad, s, W));
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
        W.q[q][k] = p < v.n ? v.xt[u64(p / kTile) * (DP * kTile) + k * kTile + p % kTile] : 0.0f;
    }
    if (lane < QW) {
        const u32 p = p0 + lane;
        W.thr[lane] = p < v.n ? thr0 : -1.0f;
        W.own[lane] = p < v.n ? v.id[p] : 0xffffffffu;
    }
    __syncwarp();
    for (u32 k = lane; k < DP; k += 32) {
        f32 lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (u32 q = 0; q < QW; ++q)
            if (p0 + q < v.n) {
                const f32 x = W.q[q][k];
                lo = x == x ? fminf(lo, x) : -INFINITY;   // (a NaN: unbounded, as in a tile's box)
                hi = x == x ? fmaxf(hi, x) : INFINITY;
            }
        W.lo[k] = lo;
        W.hi[k] = hi;
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

template <int KIND, int DP, int CH, int QW>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_knn(View v, u32 k, u32* __restrict__ ids, f32* __restrict__ dists) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, QW> sw[kWarps];
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
    walk<KIND, DP, CH, QW>(v, W, p0 / kTile, [&](u32, const f32(&c)[DP], u32 cid) -> bool {
        bool dropped = false;
#pragma unroll 1
        for (u32 q = 0; q < QW; ++q) {
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
            if (lane == 0) W.thr[q] = bound_of<KIND>(__uint_as_float(u32(kth >> 32)));
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

struct SkipComp {
    const u32* tcomp;
    const u32* scomp;
    u32 comp;   // the queries' shared component, or kNoComp
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
    }
    __syncwarp();
    const u32 first = __ballot_sync(0xffffffffu, mypos != 0xffffffffu);   // never empty: lists start groups with a query
    const u32 p_home = __shfl_sync(0xffffffffu, mypos, __ffs(first) - 1);
    const u32 c_home = __shfl_sync(0xffffffffu, mycomp, __ffs(first) - 1);
    const bool one = __all_sync(0xffffffffu, mypos == 0xffffffffu || mycomp == c_home);
#pragma unroll 1
    for (u32 e = lane; e < QW * DP; e += 32) {
        const u32 q = e / DP, k = e % DP;
        const u32 p = W.own[q] != 0xffffffffu ? qlist[g0 + q] : p_home;   // (a missing query repeats the first)
        W.q[q][k] = v.xt[u64(p / kTile) * (DP * kTile) + k * kTile + p % kTile];
    }
    __syncwarp();
    for (u32 k = lane; k < DP; k += 32) {
        f32 lo = INFINITY, hi = -INFINITY;
#pragma unroll
        for (u32 q = 0; q < QW; ++q) {
            const f32 x = W.q[q][k];
            lo = x == x ? fminf(lo, x) : -INFINITY;
            hi = x == x ? fmaxf(hi, x) : INFINITY;
        }
        W.lo[k] = lo;
        W.hi[k] = hi;
    }
    __syncwarp();
    const SkipComp skip{tcomp, scomp, one ? c_home : kNoComp};
    walk<KIND, DP, CH, QW>(
        v, W, p_home / kTile,
        [&](u32 tile, const f32(&c)[DP], u32 cid) -> bool {
            const u32 cc = __ldg(cpos + tile * kTile + lane);   // kNoComp past the points
            bool dropped = false;
#pragma unroll 1
            for (u32 q = 0; q < QW; ++q) {
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
// Row lengths (cnt by original id) and the longest row, then the rows: a
// warp collects a row's entries (id << 32 | distance bits) in shared memory,
// sorts them by id and writes the row.
template <int KIND, int DP, int CH, bool FILL>
__global__ void __launch_bounds__(32 * kWarps)
    k_near_radius(View v, f32 tau, f32 bound, u64* __restrict__ cnt, u32* __restrict__ longest,
                  const u64* __restrict__ rp, u32* __restrict__ ci, f32* __restrict__ wt) {
    pdl_wait();
    pdl_trigger();
    __shared__ WarpQ<DP, 1> sw[kWarps];
    __shared__ u64 srow[FILL ? kWarps : 1][FILL ? kRadiusRow : 1];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 p0 = blockIdx.x * kWarps + w;
    if (p0 >= v.n) return;
    WarpQ<DP, 1>& W = sw[w];
    load_queries<DP, 1>(v, p0, bound, W);
    u64* row = srow[FILL ? w : 0];
    u32 len = 0;
    walk<KIND, DP, CH, 1>(v, W, p0 / kTile, [&](u32, const f32(&c)[DP], u32 cid) -> bool {
        const f32 s = eval<KIND, DP, CH>(RegDiff<DP>{W.q[0], c});
        bool pass = cid != W.own[0] && cid != 0xffffffffu && s <= bound;
        if (!__any_sync(0xffffffffu, pass)) return false;
        const f32 d = KIND == M_L2 ? __fsqrt_rn(s) : s;
        pass = pass && d <= tau;
        const u32 m = __ballot_sync(0xffffffffu, pass);
        if constexpr (FILL) {
            const u32 o = len + __popc(m & ((1u << lane) - 1u));
            if (pass && o < kRadiusRow) row[o] = (u64(cid) << 32) | __float_as_uint(d);
        }
        len += __popc(m);
        return false;
    });
    const u32 own = W.own[0];
    if constexpr (!FILL) {
        if (lane == 0) {
            cnt[own] = len;
            if (len > kRadiusRow) atomicMax(longest, len);
        }
    } else {
        const u64 b = rp[own];
        if (len <= 32) {   // one entry a lane
            __syncwarp();
            u64 x = lane < len ? row[lane] : ~0ull;
#pragma unroll
            for (u32 size = 2; size <= 32; size <<= 1) {
#pragma unroll
                for (u32 stride = size >> 1; stride; stride >>= 1) {
                    const u64 y = __shfl_xor_sync(0xffffffffu, x, stride);
                    const bool up = ((lane & size) == 0) == ((lane & stride) == 0);
                    x = up ? (x < y ? x : y) : (x < y ? y : x);
                }
            }
            if (lane < len) {
                ci[b + lane] = u32(x >> 32);
                wt[b + lane] = __uint_as_float(u32(x));
            }
            return;
        }
        const u32 m = min(len, kRadiusRow);
        u32 P = 64;
        while (P < m) P <<= 1;
        for (u32 i = m + lane; i < P; i += 32) row[i] = ~0ull;
        __syncwarp();
        for (u32 size = 2; size <= P; size <<= 1) {
            for (u32 stride = size >> 1; stride; stride >>= 1) {
                for (u32 i = lane; i < P / 2; i += 32) {
                    const u32 lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                    const u64 x = row[lo], y = row[hi];
                    if ((x > y) == ((lo & size) == 0)) {
                        row[lo] = y;
                        row[hi] = x;
                    }
                }
                __syncwarp();
            }
        }
        for (u32 i = lane; i < m; i += 32) {
            ci[b + i] = u32(row[i] >> 32);
            wt[b + i] = __uint_as_float(u32(row[i]));
        }
    }
}

template <int KIND, int DP, int CH>
void launch_knn(tt_ctx* c, const View& v, u32 k, u32* ids, f32* dists) {
    constexpr int QW = queries_per_warp(DP);
    launch_pdl(k_near_knn<KIND, DP, CH, QW>, div_up(div_up(v.n, QW), kWarps), 32 * kWarps, 0, c->stream, v, k, ids, dists);
    TT_LAUNCH("k_near_knn");
    ++c->launches;
}

// f(padded dimension, chunks) for dim, as compile-time constants
template <int KIND, typename F>
void with_dim(u32 dim, F&& f) {
    using std::integral_constant;
    auto go = [&](auto dp, auto ch) {
        if constexpr (KIND == M_LINF) f(dp, integral_constant<int, 0>{});   // a max: no lane order
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

template <int KIND, bool FILL>
void radius_pass(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest, const u64* rp, u32* ci, f32* w) {
    // the largest eval value a kept pair can have (host copy of bound_of)
    f32 bound = tau;
    if (KIND == M_L2 && tau < INFINITY) {
        const double up = double(std::nextafter(tau, INFINITY));
        bound = std::nextafter(f32(up * up), INFINITY);
    }
    with_dim<KIND>(dim, [&](auto dp, auto ch) {
        if constexpr (decltype(dp)::value <= 8) {
            launch_pdl(k_near_radius<KIND, decltype(dp)::value, decltype(ch)::value, FILL>, div_up(v.n, kWarps),
                       32 * kWarps, 0, c->stream, v, tau, bound, cnt, longest, rp, ci, w);
            TT_LAUNCH("k_near_radius");
            ++c->launches;
        }
    });
}

template <int KIND>
void near_radius_count(tt_ctx* c, const View& v, u32 dim, f32 tau, u64* cnt, u32* longest) {
    radius_pass<KIND, false>(c, v, dim, tau, cnt, longest, nullptr, nullptr, nullptr);
}
template <int KIND>
void near_radius_fill(tt_ctx* c, const View& v, u32 dim, f32 tau, const u64* rp, u32* ci, f32* w) {
    radius_pass<KIND, true>(c, v, dim, tau, nullptr, nullptr, rp, ci, w);
}

#define TT_NEAR_INSTANTIATE(KIND)                                                     \
    template void near_knn<KIND>(tt_ctx*, const View&, u32, u32, u32*, f32*);         \
    template void near_foreign<KIND>(tt_ctx*, const View&, u32, const u32*, const u32*, const u32*, const u32*, \
                                     const u32*, u32*, unsigned long long*);          \
    template void near_radius_count<KIND>(tt_ctx*, const View&, u32, f32, u64*, u32*); \
    template void near_radius_fill<KIND>(tt_ctx*, const View&, u32, f32, const u64*, u32*, f32*);

#endif  // TT_NEAR_IMPL

}  // namespace near
}  // namespace tt
