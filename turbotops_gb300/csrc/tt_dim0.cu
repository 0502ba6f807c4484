// tt_dim0.cu — the dimension-0 stage of the cohomology reducer on the GPU.
//
// Replaces rips.hpp Reducer::dim0 (:685-870): the kept edges (d <= thr) are
// packed into Ripser-order keys and radix-sorted (the reference's bucket sort
// reproduces the plain (d asc, idx desc) order, :775-839, which is what the
// key order is); every edge gets its zero-apparent-cofacet test (:844-849,
// zero_apparent_cofacet_v :644-649); the spanning forest that the reference's
// serial union-find selects over the sorted edges (:850-866) is computed by
// Borůvka over the edge ranks — with distinct ranks the minimum spanning
// forest is unique, so the tree/non-tree split is the same edge for edge.
// H0 bars are the tree edges with d > 0 in sorted order; columns are the
// non-tree, non-apparent edges in descending order (:867).
//
// For each non-apparent edge the kernel also records the column-local part of
// the emergent-pair shortcut of compute_pairs (:903-928): the first cofacet in
// descending order with the edge's diameter, and whether that cofacet has a
// zero-apparent facet. Only the pivot lookup stays on the host.
//
// Dense complexes whose keys pack, and that keep enough of their pairs, go by vertex
// pairs (the apparent scan needs no sorted order); up to 1,280 vertices every
// count stays on the device (dim0_small), up to 91 the whole stage is one block
// (k_dim0_tiny).
//
// The same stage covers the sparse complex (rips.hpp SparseComplex :418-472):
// cofacets of an edge are the common neighbours of its endpoints, walked from
// the top of their sorted CSR rows.
#include "tt_internal.cuh"
#include "tt_rank_groups.h"

namespace tt {

namespace {

constexpr u32 NOV = 0xffffffffu;   // no vertex

// --------------------------------------------------------------------------
// Dense complex (full n x n matrix).
// --------------------------------------------------------------------------
struct DenseCx {
    const f32* mat;
    u32 n;
    __device__ __forceinline__ f32 d(u32 i, u32 j) const { return i == j ? 0.0f : mat[u64(i) * n + j]; }
};

// Largest w not in {a, b} with D[a][w] <= cap and D[b][w] <= cap, scanning
// candidates downward 32 at a time (coalesced row segments); NOV if none.
// This is the first cofacet in descending index order (cofacets_full
// rips.hpp:282-344 with all = true).
__device__ __forceinline__ u32 warp_top_cofacet2(const DenseCx& cx, u32 a, u32 b, f32 cap) {
    const int lane = threadIdx.x & 31;
    const f32* ra = cx.mat + u64(a) * cx.n;
    const f32* rb = cx.mat + u64(b) * cx.n;
    for (int64_t hi = cx.n; hi > 0; hi -= 32) {
        const int64_t w = hi - 32 + lane;
        bool ok = false;
        if (w >= 0 && u32(w) != a && u32(w) != b) ok = ra[w] <= cap && rb[w] <= cap;
        const u32 bal = __ballot_sync(0xffffffffu, ok);
        if (bal) return u32(hi - 32 + (31 - __clz(bal)));
    }
    return NOV;
}

// First facet of triangle (c0 > c1 > c2) in ascending index order with length
// d (zero_pivot_facet_v rips.hpp:609-636 for nv = 3): removing c0 leaves
// (c1, c2), removing c1 leaves (c0, c2), removing c2 leaves (c0, c1).
template <typename Cx>
__device__ __forceinline__ u64 tri_zero_facet(const Cx& cx, u32 c0, u32 c1, u32 c2, f32 d, u32& f0, u32& f1) {
    if (cx.d(c1, c2) == d) { f0 = c1; f1 = c2; return edge_idx(c1, c2); }
    if (cx.d(c0, c2) == d) { f0 = c0; f1 = c2; return edge_idx(c0, c2); }
    if (cx.d(c0, c1) == d) { f0 = c0; f1 = c1; return edge_idx(c0, c1); }
    return kNone;
}

// Rows of the complex as edge sources: row v lists its neighbours u < v in
// increasing u (the dense matrix's row prefix, or the sorted CSR row).
struct DenseRows {
    const f32* mat;
    u32 n;
    __device__ __forceinline__ u64 begin(u32) const { return 0; }
    __device__ __forceinline__ u64 end(u32 v) const { return v; }
    __device__ __forceinline__ void at(u32 v, u64 t, u32& u, f32& d) const {
        u = u32(t);
        d = mat[u64(v) * n + t];
    }
};
struct CsrRows {
    const u64* rp;
    const u32* ci;
    const f32* w;
    __device__ __forceinline__ u64 begin(u32 v) const { return rp[v]; }
    __device__ __forceinline__ u64 end(u32 v) const { return rp[v + 1]; }
    __device__ __forceinline__ void at(u32, u64 t, u32& u, f32& d) const {
        u = ci[t];
        d = w[t];
    }
};

// cnt[v] = kept edges {u, v}: u < v, d(u, v) <= thr (one warp per row);
// dmm[0] / dmm[1] = the smallest / largest distance bits kept (the sort's
// bit range, known with the count).
template <typename Rows>
__global__ void k_edge_count(Rows rows, u32 n, f32 thr, u64* __restrict__ cnt, u32* __restrict__ dmm) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const u32 warps = (gridDim.x * blockDim.x) >> 5;
    u32 lo = 0xffffffffu, hi = 0;
    for (u32 v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        const u64 b = rows.begin(v), e = rows.end(v);
        u32 c = 0;
#pragma unroll 4
        for (u64 t0 = b; t0 < e; t0 += 32) {   // (unrolled: several row loads in flight)
            bool keep = false;
            if (t0 + lane < e) {
                u32 u;
                f32 d;
                rows.at(v, t0 + lane, u, d);
                keep = u < v && d <= thr;
                if (keep) {
                    lo = min(lo, __float_as_uint(d));
                    hi = max(hi, __float_as_uint(d));
                }
            }
            c += __popc(__ballot_sync(0xffffffffu, keep));
        }
        if (lane == 0) cnt[v] = c;
    }
    // one atomic pair per block
    __shared__ u32 blo, bhi;
    if (threadIdx.x == 0) {
        blo = 0xffffffffu;
        bhi = 0;
    }
    __syncthreads();
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0 && lo <= hi) {
        atomicMin(&blo, lo);
        atomicMax(&bhi, hi);
    }
    __syncthreads();
    if (threadIdx.x == 0 && blo <= bhi) {
        atomicMin(&dmm[0], blo);
        atomicMax(&dmm[1], bhi);
    }
}

// Kept edges in a fixed order: position p = off[v] + rank in row runs over
// edge indices in increasing order (rows ascending, u ascending within a
// row). Entry q (q = m - 1 - p for the Ripser order, idx descending; q = p
// for the RedZeD order, idx ascending) gets its filtration key (DIRECT:
// packed layout), or sort key dbits << 32 | q and, beside it, idx. A stable
// sort on the dbits then yields (d, idx) in the filtration order: the ties
// keep the order of q. (m == kCountOnDevice: the count is off[n].) DIRECT saves k_edge_pack's gather and scatter by q
// (43 M edges of 12,000 points: 3.9 ms) where nothing needs the positions q.
constexpr u64 kCountOnDevice = ~0ull;
template <typename Rows, bool DIRECT>
__global__ void k_edge_fill(Rows rows, u32 n, f32 thr, const u64* __restrict__ off, u64 m, int redzed,
                            u64* __restrict__ skey, u64* __restrict__ sidx, u32* __restrict__ err) {
    pdl_wait();
    pdl_trigger();
    if (m == kCountOnDevice) m = off[n];
    const int lane = threadIdx.x & 31;
    const u32 warps = (gridDim.x * blockDim.x) >> 5;
    for (u32 v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        const u64 b = rows.begin(v), e = rows.end(v);
        const u64 vbase = u64(v) * (v - 1) / 2;
        u64 base = off[v];
#pragma unroll 4
        for (u64 t0 = b; t0 < e; t0 += 32) {
            bool keep = false;
            u32 u = 0;
            f32 d = 0.0f;
            if (t0 + lane < e) {
                rows.at(v, t0 + lane, u, d);
                keep = u < v && d <= thr;
            }
            const u32 bal = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const u64 p = base + __popc(bal & ((1u << lane) - 1));
                if (p < m) {
                    const u64 q = redzed ? p : m - 1 - p;
                    if constexpr (DIRECT) {
                        const u64 idx = vbase + u;
                        skey[q] = (u64(__float_as_uint(d)) << kIdxBits) | (redzed ? idx : kIdxMask - idx);
                    } else {
                        skey[q] = (u64(__float_as_uint(d)) << 32) | q;
                        sidx[q] = vbase + u;
                    }
                } else if (err) {
                    atomicOr(err, 1u);   // more kept edges than the caller announced
                }
            }
            base += __popc(bal);
        }
    }
}

// Sorted (dbits, q) pairs -> filtration keys (packed, or as they are in the
// wide layout, where sidx stays the index table); inv[q] = sorted position of
// the edge that index order puts at q.
__global__ void k_edge_pack(const u64* __restrict__ skey, const u64* __restrict__ sidx, u64 m, int redzed, int wide,
                            u64* __restrict__ keys, u32* __restrict__ inv) {
    pdl_wait();
    pdl_trigger();
    for (u64 r = u64(blockIdx.x) * blockDim.x + threadIdx.x; r < m; r += u64(gridDim.x) * blockDim.x) {
        const u64 k = skey[r];
        if (wide) {
            keys[r] = k;
        } else {
            const u64 idx = sidx[u32(k)];
            keys[r] = ((k >> 32) << kIdxBits) | (redzed ? idx : kIdxMask - idx);
        }
        inv[u32(k)] = u32(r);
    }
}

// The scan's result for one edge in a word: the first cofacet's vertex (NOV
// >> 2: none), whether the edge is apparent, whether the cofacet has a
// zero-apparent facet.
constexpr u32 kAppNone = NOV >> 2, kAppApparent = 1u << 30, kAppEm = 1u << 31;
constexpr u32 kAppNear = 64;    // candidates a lane tests before its warp takes the edge over
constexpr u32 kAppStep = 8;     // ... in steps (loads in flight)
constexpr u32 kAppProbe = 32;   // candidates of the emergent probe a lane tests itself

// Is there a vertex w > t, other than f0 and f1, with both lengths to f0 and
// f1 at most cap? Whole-warp scan of w in (t, hi).
__device__ __forceinline__ bool warp_any_above(const DenseCx& cx, u32 f0, u32 f1, f32 cap, u32 t, u32 hi) {
    const u32 lane = threadIdx.x & 31;
    const f32* r0 = cx.mat + u64(f0) * cx.n;
    const f32* r1 = cx.mat + u64(f1) * cx.n;
    for (int64_t top = hi; top > int64_t(t) + 1; top -= 32) {
        const int64_t w = top - 32 + lane;
        const bool ok = w > int64_t(t) && u32(w) != f0 && u32(w) != f1 && r0[w] <= cap && r1[w] <= cap;
        if (__any_sync(0xffffffffu, ok)) return true;
    }
    return false;
}

// Apparent / emergent scan of a dense complex, edge by edge in index order:
// res[idx] for every kept edge idx = (a, b), a > b.
// One warp takes 32 edges of row a (lane = b): the candidates w run down
// from n - 1, D[a][w] is one address for the warp and D[w][b] (= D[b][w], the
// matrix is symmetric bit for bit) one row segment, so an iteration tests 32
// edges with two coalesced loads from rows that all warps read (the top rows
// stay in L1 / L2). An edge of typical length has a cofacet among the first
// few candidates; the edges that none of the first kAppNear fits (short ones)
// are finished by the whole warp, 32 candidates at a time. A warp for each
// edge from the start spent its time on per-edge overhead and on random rows:
// 43 M edges of 12,000 points took 16.9 ms, this takes 5.3 (3,000 lattice
// points in R^4 under L1: 0.85 and 0.33 ms). Bound by load latency (L1 / L2).
// Beside that order there is no dependence on the sorted keys: the results
// are gathered by index when the columns are emitted.
__device__ __forceinline__ void apparent_pairs(const f32* __restrict__ mat, u32 n, f32 thr, u32 a, u32 b0,
                                               u32* __restrict__ res) {
    const DenseCx cx{mat, n};
    const u32 lane = threadIdx.x & 31, b = b0 + lane;
    {
        const f32* ra = mat + u64(a) * n;
        const u32 bl = min(b, n - 1);   // lanes past the row read in bounds
        const f32 d = b < a ? ra[b] : INFINITY;
        const bool kept = b < a && d <= thr;
        if (!__any_sync(0xffffffffu, kept)) return;
        u32 w = NOV;
        f32 da = 0.0f, db = 0.0f;   // lengths (a, w), (b, w)
        u32 hi = n;                 // candidates at and above hi are tested
        const u32 lo = n > kAppNear ? n - kAppNear : 0u;
        bool open = kept;
        while (hi > lo && __any_sync(0xffffffffu, open)) {
            f32 va[kAppStep], vb[kAppStep];
#pragma unroll
            for (u32 q = 0; q < kAppStep; ++q) {
                const u32 c = hi > q ? hi - 1 - q : 0u;
                va[q] = ra[c];
                vb[q] = mat[u64(c) * n + bl];
            }
#pragma unroll
            for (u32 q = 0; q < kAppStep; ++q) {
                const u32 c = hi - 1 - q;
                if (open && hi > q && va[q] <= d && vb[q] <= d && c != a && c != b) {
                    w = c;
                    da = va[q];
                    db = vb[q];
                    open = false;
                }
            }
            hi = hi > kAppStep ? hi - kAppStep : 0u;
        }
        // the edges still open: the whole warp, one after the other
        for (u32 rest = __ballot_sync(0xffffffffu, open); hi && rest; rest &= rest - 1) {
            const int src = __ffs(rest) - 1;
            const u32 eb = b0 + src;
            const f32 ed = __shfl_sync(0xffffffffu, d, src);
            const f32* rb = mat + u64(eb) * n;
            u32 found = NOV;
            for (int64_t top = hi; top > 0 && found == NOV; top -= 128) {
                f32 xa[4], xb[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int64_t c = top - 32 * (q + 1) + lane;
                    xa[q] = c >= 0 ? ra[c] : INFINITY;
                    xb[q] = c >= 0 ? rb[c] : INFINITY;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int64_t c = top - 32 * (q + 1) + lane;
                    const bool ok = c >= 0 && xa[q] <= ed && xb[q] <= ed && u32(c) != a && u32(c) != eb;
                    const u32 bal = __ballot_sync(0xffffffffu, ok);
                    if (found == NOV && bal) found = u32(top - 32 * (q + 1) + (31 - __clz(bal)));
                }
            }
            if (int(lane) == src && found != NOV) {
                w = found;
                da = ra[found];
                db = rb[found];
            }
        }
        // The cofacet's zero facet: the first, in ascending index order, of
        // its edges with length d (tri_zero_facet's order; (a, b) is one of
        // the three). Another edge than (a, b) only where lengths tie; the
        // emergent probe then asks whether that facet's own first cofacet is
        // this triangle, that is, whether no vertex above the third one fits.
        bool apparent = false, em = false, ask = false;
        u32 f0 = 0, f1 = 0, third = 0;
        if (kept && w != NOV) {
            u32 c0 = a, c1 = b, c2 = w;
            sort3(c0, c1, c2);
            auto len = [&](u32 u, u32 v) -> f32 {
                if (u != w && v != w) return d;
                return u == a || v == a ? da : db;
            };
            if (len(c1, c2) == d) f0 = c1, f1 = c2, third = c0;
            else if (len(c0, c2) == d) f0 = c0, f1 = c2, third = c1;
            else f0 = c0, f1 = c1, third = c2;
            apparent = f0 != w && f1 != w;
            ask = !apparent;
            em = ask;
        }
        if (__any_sync(0xffffffffu, ask)) {
            u32 c = n;   // candidates at and above c are tested
            if (ask) {
                const u32 stop = max(third + 1, n > kAppProbe ? n - kAppProbe : 0u);
                while (c > stop) {
                    --c;
                    if (c != f0 && c != f1 && mat[u64(c) * n + f0] <= d && mat[u64(c) * n + f1] <= d) {
                        em = false;
                        break;
                    }
                }
            }
            const bool more = ask && em && c > third + 1;
            for (u32 rest = __ballot_sync(0xffffffffu, more); rest; rest &= rest - 1) {
                const int src = __ffs(rest) - 1;
                const bool any = warp_any_above(cx, __shfl_sync(0xffffffffu, f0, src), __shfl_sync(0xffffffffu, f1, src),
                                                __shfl_sync(0xffffffffu, d, src), __shfl_sync(0xffffffffu, third, src),
                                                __shfl_sync(0xffffffffu, c, src));
                if (int(lane) == src) em = !any;
            }
        }
        if (kept)
            res[u64(a) * (a - 1) / 2 + b] =
                (w == NOV ? kAppNone : w) | (apparent ? kAppApparent : 0u) | (em ? kAppEm : 0u);
    }
}

__global__ void __launch_bounds__(256)
    k_apparent_pairs(const f32* __restrict__ mat, u32 n, f32 thr, u32* __restrict__ res) {
    pdl_wait();
    pdl_trigger();
    const u32 b0 = blockIdx.x * 32;
    for (u32 a = blockIdx.y * 8 + (threadIdx.x >> 5); a < n; a += gridDim.y * 8)
        if (b0 < a) apparent_pairs(mat, n, thr, a, b0, res);   // (warp-uniform)
}

// (The wide key layout, more than kPackedMaxN vertices, and thresholds that keep few
// pairs: a warp for each sorted edge, results by its sorted position.)
__global__ void k_apparent_dense(const f32* __restrict__ mat, u32 n, const u64* __restrict__ keys, EdgeFmt fmt, u64 m,
                                 u8* __restrict__ app, u32* __restrict__ emw, u8* __restrict__ emf) {
    pdl_wait();
    pdl_trigger();
    const DenseCx cx{mat, n};
    const int lane = threadIdx.x & 31;
    const u64 warps = (u64(gridDim.x) * blockDim.x) >> 5;
    for (u64 e = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; e < m; e += warps) {
        const u64 key = keys[e];
        const f32 d = fmt.d(key);
        const u64 idx = fmt.rips(key);
        u32 a, b;
        decode_edge(idx, a, b);
        const u32 w = warp_top_cofacet2(cx, a, b, d);
        bool apparent = false, em = false;
        if (w != NOV) {
            u32 c0 = a, c1 = b, c2 = w;
            sort3(c0, c1, c2);
            u32 f0 = 0, f1 = 0;
            const u64 f = tri_zero_facet(cx, c0, c1, c2, d, f0, f1);
            apparent = f == idx;
            if (!apparent) {
                // emergent probe: does the cofacet have a zero-apparent facet?
                // Its zero facet is (f0, f1); that facet's zero cofacet must
                // be the same triangle.
                const u32 w2 = warp_top_cofacet2(cx, f0, f1, d);
                if (w2 != NOV) {
                    u32 g0 = f0, g1 = f1, g2 = w2;
                    sort3(g0, g1, g2);
                    em = g0 == c0 && g1 == c1 && g2 == c2;
                }
            }
        }
        if (lane == 0) {
            app[e] = apparent;
            emw[e] = w;
            emf[e] = em;
        }
    }
}

// --------------------------------------------------------------------------
// Sparse complex (CSR, rows ascending).
// --------------------------------------------------------------------------
struct CsrCx {
    const u64* rp;
    const u32* ci;
    const f32* w;
    // Largest common neighbour x of a and b with both weights <= cap (the
    // k-way intersection walked from the top, rips.hpp:429-471), and its two
    // weights w(a, x), w(b, x).
    __device__ __forceinline__ u32 top_cofacet2(u32 a, u32 b, f32 cap, f32& wax, f32& wbx) const {
        u64 pa = rp[a + 1], pb = rp[b + 1];
        const u64 la = rp[a], lb = rp[b];
        while (pa > la && pb > lb) {
            const u32 xa = ci[pa - 1], xb = ci[pb - 1];
            if (xa > xb) { --pa; continue; }
            if (xb > xa) { --pb; continue; }
            const f32 x1 = w[pa - 1], x2 = w[pb - 1];
            if (x1 <= cap && x2 <= cap) {
                wax = x1;
                wbx = x2;
                return xa;
            }
            --pa;
            --pb;
        }
        return NOV;
    }
};

// Edges are visited in index order (inv: index order -> sorted position), so
// neighbouring threads share the larger vertex's row; results go to the
// edge's sorted position.
// (32 registers: 64 warps an SM to hide the walk's load latency.)
__global__ void __launch_bounds__(256, 8)
    k_apparent_csr(CsrCx cx, const u64* __restrict__ keys, EdgeFmt fmt, const u32* __restrict__ inv, u64 m,
                   u8* __restrict__ app, u32* __restrict__ emw, u8* __restrict__ emf) {
    pdl_wait();
    pdl_trigger();
    for (u64 t = u64(blockIdx.x) * blockDim.x + threadIdx.x; t < m; t += u64(gridDim.x) * blockDim.x) {
        const u64 e = inv[t];
        const u64 key = keys[e];
        const f32 d = fmt.d(key);
        const u64 idx = fmt.rips(key);
        u32 a, b;
        decode_edge(idx, a, b);
        f32 wax = 0.0f, wbx = 0.0f;
        const u32 w = cx.top_cofacet2(a, b, d, wax, wbx);
        bool apparent = false, em = false;
        if (w != NOV) {
            u32 c0 = a, c1 = b, c2 = w;
            sort3(c0, c1, c2);
            // the zero facet (tri_zero_facet's order) from the three known
            // edge lengths: (a, b) = d, (a, w) = wax, (b, w) = wbx
            auto len = [&](u32 u, u32 v) -> f32 {
                if ((u == a && v == b) || (u == b && v == a)) return d;
                return u == a || v == a ? wax : wbx;
            };
            u32 f0, f1;
            if (len(c1, c2) == d) f0 = c1, f1 = c2;
            else if (len(c0, c2) == d) f0 = c0, f1 = c2;
            else f0 = c0, f1 = c1;   // (a, b) is one of the three pairs: one length equals d
            apparent = edge_idx(f0, f1) == idx;
            if (!apparent) {
                f32 t1, t2;
                const u32 w2 = cx.top_cofacet2(f0, f1, d, t1, t2);
                if (w2 != NOV) {
                    u32 g0 = f0, g1 = f1, g2 = w2;
                    sort3(g0, g1, g2);
                    em = g0 == c0 && g1 == c1 && g2 == c2;
                }
            }
        }
        app[e] = apparent;
        emw[e] = w;
        emf[e] = em;
    }
}

// --------------------------------------------------------------------------
// Borůvka over edge ranks (rank = position in the sorted array).
// --------------------------------------------------------------------------
__global__ void k_iota(u32* __restrict__ p, u32 n) {
    pdl_wait();
    pdl_trigger();
    for (u32 v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) p[v] = v;
}

// For each live edge with endpoints in different components, offer its rank
// to both components; edges inside a component are dropped from the list.
// A round's edges are the survivors of the rounds before (`live`, their count
// read from the previous round's counter, so rounds run without a host round
// trip) and the sorted edges [lo, hi) that join in this round. (The
// survivors' list grows by one atomic per warp: ranks from a ballot.)
// A component's best rank only falls, so an offer that a plain load already
// shows to be too large is not issued: the largest component receives most of
// the edges, and their atomics on its one word were most of the forest's time
// (43 M edges of 12,000 points: 23 ms a round).
__global__ void k_bv_offer(const u64* __restrict__ keys, EdgeFmt fmt, const u32* __restrict__ live,
                           const u32* __restrict__ nlive_in, u32 lo, u32 hi, const u32* __restrict__ comp,
                           u32* best, u32* __restrict__ live_out, u32* __restrict__ nlive_out) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31;
    const u64 nlive = nlive_in ? *nlive_in : 0u;
    const u64 total = nlive + (hi - lo);
    for (u64 base = u64(blockIdx.x) * blockDim.x; base < total; base += u64(gridDim.x) * blockDim.x) {
        const u64 t = base + threadIdx.x;   // whole warps iterate together
        bool keep = false;
        u32 r = 0;
        if (t < total) {
            r = t < nlive ? live[t] : lo + u32(t - nlive);
            u32 a, b;
            decode_edge(fmt.rips(keys[r]), a, b);
            const u32 ca = comp[a], cb = comp[b];
            if (ca != cb) {
                if (*reinterpret_cast<volatile const u32*>(best + ca) > r) atomicMin(&best[ca], r);
                if (*reinterpret_cast<volatile const u32*>(best + cb) > r) atomicMin(&best[cb], r);
                keep = true;
            }
        }
        const u32 m = __ballot_sync(0xffffffffu, keep);
        if (!m) continue;
        u32 pos = 0;
        if (lane == u32(__ffs(m) - 1)) pos = atomicAdd(nlive_out, u32(__popc(m)));
        pos = __shfl_sync(0xffffffffu, pos, __ffs(m) - 1);
        if (keep) live_out[pos + __popc(m & ((1u << lane) - 1u))] = r;
    }
}

// Every component root with an offered edge takes it into the forest and
// hooks onto the other side; of a mutual pair only the larger root hooks.
// (The hook count is summed per warp: one atomic a warp. A round whose offer
// found no edge between components has nothing to hook: live == 0.)
__global__ void k_bv_hook(const u64* __restrict__ keys, EdgeFmt fmt, const u32* __restrict__ comp,
                          const u32* __restrict__ best,
                          u32* __restrict__ parent, u8* __restrict__ tree, u32 n, u32* __restrict__ hooks,
                          const u32* __restrict__ live) {
    pdl_wait();
    pdl_trigger();
    if (*live == 0) return;
    u32 mine = 0;
    for (u32 c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        if (comp[c] != c) continue;
        const u32 r = best[c];
        if (r == NOV) continue;
        u32 a, b;
        decode_edge(fmt.rips(keys[r]), a, b);
        const u32 o = comp[a] == c ? comp[b] : comp[a];
        tree[r] = 1;
        if (best[o] == r && c < o) continue;   // mutual: o hooks onto c
        parent[c] = o;
        ++mine;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(hooks, mine);
}

__global__ void k_bv_flatten(const u32* __restrict__ parent, u32* __restrict__ comp, u32* __restrict__ best, u32 n,
                             const u32* __restrict__ live) {
    pdl_wait();
    pdl_trigger();
    if (*live == 0) return;   // no hook this round: parents, components and offers unchanged
    for (u32 v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        u32 r = parent[v];
        for (u32 s = 0; parent[r] != r && s < n; ++s) r = parent[r];
        comp[v] = r;
        best[v] = NOV;
    }
}

// --------------------------------------------------------------------------
// Ordered compaction of H0 bars and columns.
// --------------------------------------------------------------------------
// Two passes over the sorted edges: counts per run of kRun edges (one warp a
// run), a scan of the counts, then the emit with the ranks inside a run from
// ballots. (Per-edge flag and offset words instead cost 32 bytes an edge of
// traffic; what bounds the pair form's count now is its 4-byte gather by
// edge index, 1.1 ms for 43 M edges; the emit takes 0.23.)
// PAIRS: the apparent scan's results are k_apparent_pairs' words by edge
// index, and the count pass writes the per-edge apparent flags from them;
// otherwise they are per-edge arrays in sorted order.
constexpr u32 kRun = 512;

// cnt[run] = finite H0 bars << 32 | columns.
template <bool PAIRS>
__global__ void k_count_dim0(const u64* __restrict__ keys, EdgeFmt fmt, const u8* __restrict__ tree, u8* __restrict__ app,
                             const u32* __restrict__ res, u64 m, const u64* __restrict__ mdev, int want_cols,
                             u64* __restrict__ cnt) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31;
    const u64 cap_runs = (m + kRun - 1) / kRun;   // runs past the count get zeros (the scan covers the capacity)
    if (mdev) m = *mdev;
    const u64 runs = (m + kRun - 1) / kRun;
    const u64 warps = (u64(gridDim.x) * blockDim.x) >> 5;
    for (u64 run = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; run < cap_runs; run += warps) {
        if (run >= runs) {
            if (lane == 0) cnt[run] = 0;
            continue;
        }
        u32 h = 0, cols = 0;
#pragma unroll 4
        for (u32 i = 0; i < kRun; i += 32) {
            const u64 e = run * kRun + i + lane;
            if (e >= m) continue;
            const u64 key = keys[e];
            const bool t = tree[e];
            h += t && fmt.d(key) > 0.0f;
            if (want_cols) {
                bool ap;
                if constexpr (PAIRS) {
                    ap = (res[fmt.rips(key)] & kAppApparent) != 0;
                    app[e] = ap;
                } else {
                    ap = app[e];
                }
                cols += !t && !ap;
            }
        }
        h = __reduce_add_sync(0xffffffffu, h);
        cols = __reduce_add_sync(0xffffffffu, cols);
        if (lane == 0) cnt[run] = (u64(h) << 32) | cols;
    }
}

// off: the exclusive scan of cnt (m < 2^32: one sum counts both without a
// carry between the halves), tot its total.
template <bool PAIRS>
__global__ void k_emit_dim0(const u64* __restrict__ keys, EdgeFmt fmt, const u8* __restrict__ tree,
                            const u8* __restrict__ app, const u32* __restrict__ emw, const u8* __restrict__ emf, u64 m,
                            const u64* __restrict__ mdev, int want_cols, const u64* __restrict__ off, const u64* __restrict__ tot,
                            f32* __restrict__ h0, u64* __restrict__ h0_edge, u64* __restrict__ cidx,
                            f32* __restrict__ cd, u64* __restrict__ emi, u8* __restrict__ emf_out) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    if (mdev) m = *mdev;
    const u64 ncols = tot[0] & 0xffffffffull;
    const u64 runs = (m + kRun - 1) / kRun;
    const u64 warps = (u64(gridDim.x) * blockDim.x) >> 5;
    for (u64 run = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; run < runs; run += warps) {
        u64 oh = off[run] >> 32, oc = off[run] & 0xffffffffull;
#pragma unroll 4
        for (u32 i = 0; i < kRun; i += 32) {
            const u64 e = run * kRun + i + lane;
            const bool in = e < m;
            const bool t = in && tree[e];
            const bool col = in && want_cols && !t && !app[e];
            const u64 key = in ? keys[e] : 0ull;
            const f32 d = fmt.d(key);
            const bool bar = t && d > 0.0f;
            const u32 hb = __ballot_sync(0xffffffffu, bar), cb = __ballot_sync(0xffffffffu, col);
            if (bar) {
                const u64 o = oh + __popc(hb & lt);
                h0[o] = d;
                h0_edge[o] = fmt.rips(key);   // the bar's critical (death) edge
            }
            if (col) {
                const u64 o = ncols - 1 - (oc + __popc(cb & lt));   // descending order (rips.hpp:867)
                const u64 idx = fmt.rips(key);
                cidx[o] = idx;
                cd[o] = d;
                u32 w;
                u8 em;
                if constexpr (PAIRS) {
                    const u32 r = emw[idx];
                    w = (r & kAppNone) == kAppNone ? NOV : r & kAppNone;
                    em = (r & kAppEm) != 0;
                } else {
                    w = emw[e];
                    em = emf[e];
                }
                if (w == NOV) {
                    emi[o] = kNone;
                    emf_out[o] = 0;
                } else {
                    u32 a, b;
                    decode_edge(idx, a, b);
                    u32 c0 = a, c1 = b, c2 = w;
                    sort3(c0, c1, c2);
                    emi[o] = tri_idx(c0, c1, c2);
                    emf_out[o] = em;
                }
            }
            oh += __popc(hb);
            oc += __popc(cb);
        }
    }
}


// --------------------------------------------------------------------------
// The spanning forest of a small dense complex (n <= kSmallN) without a host
// round trip: one block runs the Boruvka rounds on the shortest edges with
// the components in shared memory, a filter keeps the later edges that still
// join two components (usually none: the forest is complete), and the block
// finishes with those. (The rounds of separate kernels cost three launches
// and a share of a round trip each, whatever the size.)
// --------------------------------------------------------------------------
// (Up to 1,280: with the sort on the capacity's worth of keys instead of the kept
// ones and one block for the forest, the stage is the slower one from there on.
// Gaussian points in R^3, this / the separate rounds in us, 1/64 of the pairs kept
// and up to the enclosing radius: 600 points 141 / 199 and 200 / 249, 1,200 223 / 235
// and 416 / 361, 1,500 251 / 237 and 511 / 385, 2,048 331 / 263 and 1,105 / 471.)
constexpr u32 kSmallN = 1280;
constexpr u32 kForestThreads = 1024;

// Edges: the ranks [0, min(*m, first)) when `first`, else list[0, *count).
// st[0] = hooks so far, st[1] = live edges (the filter's list).
__global__ void __launch_bounds__(kForestThreads) k_forest_block(const u64* __restrict__ keys, const u64* __restrict__ m,
                                                                u32 first, const u32* __restrict__ list, u32 n,
                                                                u32* __restrict__ comp_g, u8* __restrict__ tree,
                                                                u32* __restrict__ st) {
    pdl_wait();
    pdl_trigger();
    __shared__ u32 comp[kSmallN], parent[kSmallN], best[kSmallN];
    __shared__ u32 hooked;
    const u32 tid = threadIdx.x;
    const u32 before = first ? 0u : st[0];
    const u32 cnt = first ? u32(min(*m, u64(first))) : st[1];
    if (!first && cnt == 0) return;
    for (u32 v = tid; v < n; v += kForestThreads) {
        const u32 c = first ? v : comp_g[v];
        comp[v] = parent[v] = c;
        best[v] = NOV;
    }
    if (tid == 0) hooked = 0;
    __syncthreads();
    const EdgeFmt fmt{};
    for (;;) {
        bool any = false;
        for (u32 e = tid; e < cnt; e += kForestThreads) {
            const u32 r = first ? e : list[e];
            u32 a, b;
            decode_edge(fmt.rips(keys[r]), a, b);
            const u32 ca = comp[a], cb = comp[b];
            if (ca == cb) continue;
            any = true;
            if (*reinterpret_cast<volatile u32*>(&best[ca]) > r) atomicMin(&best[ca], r);
            if (*reinterpret_cast<volatile u32*>(&best[cb]) > r) atomicMin(&best[cb], r);
        }
        if (!__syncthreads_or(any)) break;
        for (u32 c = tid; c < n; c += kForestThreads) {
            const u32 r = best[c];
            if (comp[c] != c || r == NOV) continue;
            u32 a, b;
            decode_edge(fmt.rips(keys[r]), a, b);
            const u32 o = comp[a] == c ? comp[b] : comp[a];
            tree[r] = 1;
            if (best[o] == r && c < o) continue;   // mutual: o hooks onto c
            parent[c] = o;
            atomicAdd(&hooked, 1u);
        }
        __syncthreads();
        for (u32 v = tid; v < n; v += kForestThreads) {
            u32 r = parent[comp[v]];
            for (u32 q = 0; parent[r] != r && q < n; ++q) r = parent[r];
            comp[v] = r;
        }
        __syncthreads();
        for (u32 v = tid; v < n; v += kForestThreads) {
            parent[v] = comp[v];
            best[v] = NOV;
        }
        __syncthreads();
        if (before + hooked == n - 1) break;   // (shared, read after a barrier and next written after one)
    }
    __syncthreads();
    for (u32 v = tid; v < n; v += kForestThreads) comp_g[v] = comp[v];
    if (tid == 0) st[0] = before + hooked;
}

// The edges [first, *m) that join two components, unless the forest is
// complete: list[0, st[1]).
__global__ void k_forest_filter(const u64* __restrict__ keys, const u64* __restrict__ m, u32 first, u32 n,
                                const u32* __restrict__ comp, u32* __restrict__ list, u32* __restrict__ st) {
    pdl_wait();
    pdl_trigger();
    if (st[0] == n - 1) return;
    const u32 lane = threadIdx.x & 31;
    const u64 total = *m;
    const EdgeFmt fmt{};
    for (u64 base = first + u64(blockIdx.x) * blockDim.x; base < total; base += u64(gridDim.x) * blockDim.x) {
        const u64 r = base + threadIdx.x;   // whole warps iterate together
        bool keep = false;
        if (r < total) {
            u32 a, b;
            decode_edge(fmt.rips(keys[r]), a, b);
            keep = comp[a] != comp[b];
        }
        const u32 bal = __ballot_sync(0xffffffffu, keep);
        if (!bal) continue;
        u32 pos = 0;
        if (lane == 0) pos = atomicAdd(st + 1, u32(__popc(bal)));
        pos = __shfl_sync(0xffffffffu, pos, 0);
        if (keep) list[pos + __popc(bal & ((1u << lane) - 1u))] = u32(r);
    }
}

// --------------------------------------------------------------------------
// The whole stage of a tiny dense complex (n <= kTinyN) in one block: the kept
// edges' keys in shared memory, ordered by a bitonic sort (the keys are
// distinct and their order total), the apparent scan, the spanning forest, and
// the outputs with the counts of what is kept into page-locked memory. A cloud
// of 64 points is then one launch and one wait (with the stages as kernels of
// their own, about twenty launches of 2 to 4 us: 155 us a pass with its
// matrix and the copies of its results; now 110).
// --------------------------------------------------------------------------
// (Up to 91: 4,095 pairs, a bitonic sort of 4,096. 91 points 110 us, dim0_small's
// kernels 112; 92 points, sorting 8,192, 148 and 116; 128 points 238 and 116.)
constexpr u32 kTinyN = 91;
constexpr u32 kTinyPairs = kTinyN * (kTinyN - 1) / 2;   // 4,095
constexpr u32 kTinyKeys = 4096;
constexpr u32 kTinyThreads = 1024;
struct TinySmem {
    u64 key[kTinyKeys];
    u32 res[kTinyPairs];
    u8 tree[kTinyKeys];
    u32 comp[kTinyN], parent[kTinyN], best[kTinyN];
    u32 warp[kTinyThreads / 32];
    u32 hooked;
};

__global__ void __launch_bounds__(kTinyThreads)
    k_dim0_tiny(const f32* __restrict__ mat, u32 n, f32 thr, int want_cols, u64* __restrict__ keys,
                u8* __restrict__ app, u8* __restrict__ tree, f32* __restrict__ h0, u64* __restrict__ h0_edge,
                u64* __restrict__ cidx, f32* __restrict__ cd, u64* __restrict__ emi, u8* __restrict__ emf,
                u64* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char tiny_raw[];
    TinySmem& S = *reinterpret_cast<TinySmem*>(tiny_raw);
    const u32 tid = threadIdx.x, lane = tid & 31, w = tid >> 5, lt = (1u << lane) - 1u;
    const u32 pairs = n * (n - 1) / 2;
    u32 P = 2;
    while (P < pairs) P <<= 1;
    const EdgeFmt fmt{};
    // keys of the kept edges, the rest after every key
    u32 m = 0;
    for (u32 e0 = 0; e0 < P; e0 += kTinyThreads) {
        const u32 e = e0 + tid;
        bool keep = false;
        if (e < P) {
            u64 k = ~0ull;
            if (e < pairs) {
                u32 a, b;
                decode_edge(e, a, b);
                const f32 d = mat[a * n + b];
                keep = d <= thr;
                if (keep) k = key_rips(d, e);
            }
            S.key[e] = k;
            S.tree[e] = 0;
        }
        m += __syncthreads_count(keep);
    }
    if (tid < n) {
        S.comp[tid] = S.parent[tid] = tid;
        S.best[tid] = NOV;
    }
    if (tid == 0) S.hooked = 0;
    if (want_cols)   // (row, 32 columns) tasks, a warp each
        for (u32 t = w, chunks = (n + 31) / 32; t < n * chunks; t += kTinyThreads / 32) {
            const u32 a = t / chunks, b0 = t % chunks * 32;
            if (b0 < a) apparent_pairs(mat, n, thr, a, b0, S.res);
        }
    __syncthreads();
    for (u32 size = 2; size <= P; size <<= 1)
        for (u32 stride = size >> 1; stride; stride >>= 1) {
            for (u32 i = tid; i < P / 2; i += kTinyThreads) {
                const u32 lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const u64 x = S.key[lo], y = S.key[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    S.key[lo] = y;
                    S.key[hi] = x;
                }
            }
            __syncthreads();
        }
    // the spanning forest (k_forest_block's rounds)
    for (;;) {
        bool any = false;
        for (u32 r = tid; r < m; r += kTinyThreads) {
            u32 a, b;
            decode_edge(fmt.rips(S.key[r]), a, b);
            const u32 ca = S.comp[a], cb = S.comp[b];
            if (ca == cb) continue;
            any = true;
            if (*reinterpret_cast<volatile u32*>(&S.best[ca]) > r) atomicMin(&S.best[ca], r);
            if (*reinterpret_cast<volatile u32*>(&S.best[cb]) > r) atomicMin(&S.best[cb], r);
        }
        if (!__syncthreads_or(any)) break;
        if (tid < n && S.comp[tid] == tid && S.best[tid] != NOV) {
            const u32 r = S.best[tid];
            u32 a, b;
            decode_edge(fmt.rips(S.key[r]), a, b);
            const u32 o = S.comp[a] == tid ? S.comp[b] : S.comp[a];
            S.tree[r] = 1;
            if (!(S.best[o] == r && tid < o)) {   // mutual: o hooks onto this one
                S.parent[tid] = o;
                atomicAdd(&S.hooked, 1u);
            }
        }
        __syncthreads();
        u32 root = 0;
        if (tid < n) {
            root = S.parent[S.comp[tid]];
            for (u32 q = 0; S.parent[root] != root && q < n; ++q) root = S.parent[root];
        }
        __syncthreads();
        if (tid < n) {
            S.comp[tid] = S.parent[tid] = root;
            S.best[tid] = NOV;
        }
        __syncthreads();
        if (S.hooked == n - 1) break;   // (read after a barrier, next written after one)
    }
    __syncthreads();
    // columns in all (they are written in descending order), then the outputs
    u32 ncols = 0;
    if (want_cols)
        for (u32 e0 = 0; e0 < m; e0 += kTinyThreads) {
            const u32 e = e0 + tid;
            const bool col = e < m && !S.tree[e] && !(S.res[u32(fmt.rips(S.key[e]))] & kAppApparent);
            ncols += __syncthreads_count(col);
        }
    u32 oh = 0, oc = 0;   // bars and columns before this chunk
    for (u32 e0 = 0; e0 < m; e0 += kTinyThreads) {
        const u32 e = e0 + tid;
        const bool in = e < m;
        const u64 key = in ? S.key[e] : 0ull;
        const u32 idx = u32(fmt.rips(key));
        const f32 d = fmt.d(key);
        const bool t = in && S.tree[e];
        const u32 r = in && want_cols ? S.res[idx] : 0u;
        const bool ap = (r & kAppApparent) != 0;
        const bool bar = t && d > 0.0f, col = in && want_cols && !t && !ap;
        const u32 hb = __ballot_sync(0xffffffffu, bar), cb = __ballot_sync(0xffffffffu, col);
        __syncthreads();   // the last chunk's counts are read
        if (lane == 0) S.warp[w] = (u32(__popc(hb)) << 16) | __popc(cb);
        __syncthreads();
        u32 before = 0, all = 0;   // bars << 16 | columns (at most 1,024 each)
#pragma unroll
        for (u32 q = 0; q < kTinyThreads / 32; ++q) {
            const u32 x = S.warp[q];
            before += q < w ? x : 0u;
            all += x;
        }
        if (in) {
            keys[e] = key;
            tree[e] = t;
            if (want_cols) app[e] = ap;
        }
        if (bar) {
            const u32 o = oh + (before >> 16) + __popc(hb & lt);
            h0[o] = d;
            h0_edge[o] = idx;
        }
        if (col) {
            const u32 o = ncols - 1 - (oc + (before & 0xffffu) + __popc(cb & lt));
            cidx[o] = idx;
            cd[o] = d;
            const u32 cw = r & kAppNone;
            if (cw == kAppNone) {
                emi[o] = kNone;
                emf[o] = 0;
            } else {
                u32 c0, c1, c2 = cw;
                decode_edge(idx, c0, c1);
                sort3(c0, c1, c2);
                emi[o] = tri_idx(c0, c1, c2);
                emf[o] = (r & kAppEm) != 0;
            }
        }
        oh += all >> 16;
        oc += all & 0xffffu;
    }
    if (tid == 0) {
        status[0] = (u64(oh) << 32) | oc;
        status[1] = S.hooked;
        status[2] = m;
    }
}

inline u32 grid_for(u64 work, u32 per_block) {
    const u64 g = (work + per_block - 1) / per_block;
    return u32(std::max<u64>(1, std::min<u64>(g, 64ull * kSMs)));
}

}  // namespace

// Kept edges as sorted keys (Ripser or RedZeD order); returns the count.
// The edges are written in index order (count, scan, fill), so one stable
// sort on the distance bits alone gives the filtration order: only the bits
// in which the kept distances differ (their range comes back with the count),
// three passes when 25 bits differ, instead of a full 64-bit key sort.
// Slots: S_EDGE_CNT, S_EDGE_SORT, S_EDGE_IDX, S_EDGE_KEYS (result),
// S_EDGE_INV (result: index order -> sorted position),
// and the sort's own (S_SORT_A, S_SORT_HIST, S_SCAN*, S_MISC3).
// Above kPackedMaxN vertices the keys take the wide layout (EdgeFmt) and
// *eidx_out the index table; otherwise *eidx_out is null. m_known (not
// kUnknownM): the caller knows the kept-edge count (a symmetric graph without
// self loops cut at +inf keeps nnz / 2), so the count is not read back: the
// sort takes all 31 distance bits, and a wrong count sets *err instead of
// writing out of bounds.
constexpr u64 kUnknownM = ~0ull;
// want_inv: S_EDGE_INV is needed (k_apparent_csr walks the edges in index
// order); without it, packed keys are written by the fill itself.
static u64 sorted_edge_keys(tt_ctx* c, const Complex& cx, int redzed, bool want_inv, u64** keys_out, u64** eidx_out,
                            u64 m_known = kUnknownM, u32* err = nullptr) {
    const u32 n = cx.n;
    u64 m = 0;
    u64* off = c->arena.get<u64>(S_EDGE_CNT, u64(n) + 2);
    u32* dmm = reinterpret_cast<u32*>(off + n + 1);   // beside the total: one copy brings both
    const u32 g = grid_for(u64(n) * 32, 256);
    int dbits = 0;   // distance bits the sort must see
    if (n > 1) {
        TT_CUDA(cudaMemsetAsync(dmm, 0xff, sizeof(u32), c->stream));
        TT_CUDA(cudaMemsetAsync(dmm + 1, 0, sizeof(u32), c->stream));
        if (cx.mat)
            launch_pdl(k_edge_count<DenseRows>, g, 256, 0, c->stream, DenseRows{cx.mat, n}, n, cx.thr, off, dmm);
        else
            launch_pdl(k_edge_count<CsrRows>, g, 256, 0, c->stream, CsrRows{cx.rp, cx.ci, cx.w}, n, cx.thr, off, dmm);
        TT_LAUNCH("k_edge_count");
        ++c->launches;
        scan_exclusive<u64>(c, off, off, n, off + n);
        if (m_known != kUnknownM) {
            m = m_known;
            dbits = 31;   // every bit of a non-negative float: the same three passes
        } else {
            u64 h[2];
            TT_CUDA(cudaMemcpyAsync(h, off + n, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
            TT_CUDA(cudaStreamSynchronize(c->stream));
            m = h[0];
            const u32 lo = u32(h[1]), hi = u32(h[1] >> 32);
            const u32 diff = m ? lo ^ hi : 0u;
            dbits = diff ? 32 - __builtin_clz(diff) : 0;
        }
    }
    if (m >= 0xffffffffull) invalid("gb300: more than 2^32 - 1 kept edges");
    u64* keys = c->arena.get<u64>(S_EDGE_KEYS, m + 1);
    const bool wide = n > kPackedMaxN;
    const bool direct = !wide && !want_inv;
    *eidx_out = nullptr;
    if (m) {
        u64* kb = c->arena.get<u64>(S_SORT_A, m);
        // direct: filled into whichever buffer the sort's passes bring back to `keys`
        const bool odd = radix_passes(m, dbits) & 1;
        u64* skey = !direct ? c->arena.get<u64>(S_EDGE_SORT, m + 1) : odd ? kb : keys;
        u64* sidx = direct ? nullptr : c->arena.get<u64>(S_EDGE_IDX, m + 1);
        auto fill = [&](auto rows, auto dir) {
            launch_pdl(k_edge_fill<decltype(rows), decltype(dir)::value>, g, 256, 0, c->stream, rows, n, cx.thr, off, m,
                       redzed, skey, sidx, err);
        };
        auto fill_rows = [&](auto rows) {
            if (direct) fill(rows, std::true_type{});
            else fill(rows, std::false_type{});
        };
        if (cx.mat) fill_rows(DenseRows{cx.mat, n});
        else fill_rows(CsrRows{cx.rp, cx.ci, cx.w});
        TT_LAUNCH("k_edge_fill");
        // a stable sort on the distance bits that differ (none: already in order)
        const bool sw = dbits > 0 && radix_sort<u32>(c, skey, static_cast<u32*>(nullptr), m, direct && odd ? keys : kb,
                                                     static_cast<u32*>(nullptr), dbits, direct ? kIdxBits : 32);
        c->launches += 1;
        if (!direct) {
            u32* inv = c->arena.get<u32>(S_EDGE_INV, m + 1);
            launch_pdl(k_edge_pack, grid_for(m, 256), 256, 0, c->stream, sw ? kb : skey, sidx, m, redzed, wide, keys, inv);
            if (wide) *eidx_out = sidx;
            TT_LAUNCH("k_edge_pack");
            c->launches += 1;
        }
    }
    *keys_out = keys;
    return m;
}

// dim0 of a dense complex of at most kSmallN vertices: the same stages, every
// buffer at its largest size and every count left on the device, so that the
// host waits once, at the end (sizes of a few hundred points spent most of
// their time in round trips and launches).
static void dim0_small(tt_ctx* c, const Complex& cx, u32 maxdim, Dim0Out& out) {
    const u32 n = cx.n;
    const u64 cap = u64(n) * (n - 1) / 2;
    const int want_cols = maxdim >= 1;
    const cudaStream_t s = c->stream;
    u64* off = c->arena.get<u64>(S_EDGE_CNT, u64(n) + 2);
    const u64* mdev = off + n;
    u32* dmm = reinterpret_cast<u32*>(off + n + 1);
    u64* keys = c->arena.get<u64>(S_EDGE_KEYS, cap + 1);
    u64* kb = c->arena.get<u64>(S_SORT_A, cap);
    u8* app = c->arena.get<u8>(S_FLAGS, 2 * cap + 16);
    u8* tree = app + cap + 8;
    u32* res = c->arena.get<u32>(S_EDGE_TMP, cap + 1);
    u32* comp = c->arena.get<u32>(S_UF_PARENT, n);
    u32* list = c->arena.get<u32>(S_UF_WORK, cap + 1);
    const u64 runs = (cap + kRun - 1) / kRun;
    u64* cnt = c->arena.get<u64>(S_MISC0, runs + 1);
    u64* tot = c->arena.get<u64>(S_COUNT, 4);
    u32* st = reinterpret_cast<u32*>(tot + 1);
    out.keys = keys;
    out.app = want_cols ? app : nullptr;
    out.tree = tree;
    out.h0 = c->arena.get<f32>(S_OUT0, n + 1);
    out.cidx = c->arena.get<u64>(S_OUT1, (want_cols ? cap : 0) + 1);
    out.cd = c->arena.get<f32>(S_OUT2, (want_cols ? cap : 0) + 1);
    out.emi = c->arena.get<u64>(S_OUT3, (want_cols ? cap : 0) + 1);
    out.emf = c->arena.get<u8>(S_OUT4, (want_cols ? cap : 0) + 1);
    out.h0_edge = c->arena.get<u64>(S_OUT5, n + 1);
    u64* h = static_cast<u64*>(c->pinned.get(4 * sizeof(u64)));
    auto finish = [&] {
        TT_CUDA(cudaStreamSynchronize(s));
        out.m = h[2];
        out.nh0 = h[0] >> 32;
        out.ncols = h[0] & 0xffffffffull;
        out.essential = n - u32(h[1]);
    };
    if (n <= kTinyN) {
        TT_CUDA(cudaFuncSetAttribute(k_dim0_tiny, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TinySmem))));
        k_dim0_tiny<<<1, kTinyThreads, sizeof(TinySmem), s>>>(cx.mat, n, cx.thr, want_cols, keys, app, tree, out.h0,
                                                              out.h0_edge, out.cidx, out.cd, out.emi, out.emf, h);
        TT_LAUNCH("k_dim0_tiny");
        c->launches += 1;
        finish();
        return;
    }
    const EdgeFmt fmt{};
    TT_CUDA(cudaMemsetAsync(tot, 0, 4 * sizeof(u64), s));
    TT_CUDA(cudaMemsetAsync(tree, 0, cap + 1, s));
    // the apparent scan beside the sort and the forest, once it is long enough
    // to pay for the fork
    SideScope side(c);
    if (want_cols) {
        const cudaStream_t as = n > 512 ? side.fork() : s;
        launch_pdl(k_apparent_pairs, dim3(div_up(n, 32), div_up(n, 8)), 256, 0, as, cx.mat, n, cx.thr, res);
        TT_LAUNCH("k_apparent");
        ++c->launches;
    }
    const u32 g = grid_for(u64(n) * 32, 256);
    launch_pdl(k_edge_count<DenseRows>, g, 256, 0, s, DenseRows{cx.mat, n}, n, cx.thr, off, dmm);
    TT_LAUNCH("k_edge_count");
    scan_exclusive<u64>(c, off, off, n, off + n);
    constexpr int kBits = 31;   // every bit of a non-negative float: as many passes as 23 bits
    const bool odd = radix_passes(cap, kBits) & 1;
    launch_pdl(k_edge_fill<DenseRows, true>, g, 256, 0, s, DenseRows{cx.mat, n}, n, cx.thr, off, kCountOnDevice, 0,
               odd ? kb : keys, static_cast<u64*>(nullptr), static_cast<u32*>(nullptr));
    TT_LAUNCH("k_edge_fill");
    radix_sort<u32>(c, odd ? kb : keys, static_cast<u32*>(nullptr), cap, odd ? keys : kb, static_cast<u32*>(nullptr),
                    kBits, kIdxBits, reinterpret_cast<const unsigned long long*>(mdev));
    const u32 first = std::max<u32>(8 * n, 4 * kForestThreads);
    launch_pdl(k_forest_block, 1, kForestThreads, 0, s, keys, mdev, first, list, n, comp, tree, st);
    TT_LAUNCH("k_forest_block");
    c->launches += 3;
    if (cap > first) {
        launch_pdl(k_forest_filter, grid_for(cap - first, 256), 256, 0, s, keys, mdev, first, n,
                   static_cast<const u32*>(comp), list, st);
        TT_LAUNCH("k_forest_filter");
        launch_pdl(k_forest_block, 1, kForestThreads, 0, s, keys, mdev, 0u, list, n, comp, tree, st);
        TT_LAUNCH("k_forest_block");
        c->launches += 2;
    }
    side.join();
    const u32 gr = grid_for(runs * 32, 256);
    launch_pdl(k_count_dim0<true>, gr, 256, 0, s, keys, fmt, tree, app, res, cap, mdev, want_cols, cnt);
    TT_LAUNCH("k_count_dim0");
    scan_exclusive<u64>(c, cnt, cnt, runs, tot);
    launch_pdl(k_emit_dim0<true>, gr, 256, 0, s, keys, fmt, tree, app, res, static_cast<const u8*>(nullptr), cap, mdev,
               want_cols, cnt, tot, out.h0, out.h0_edge, out.cidx, out.cd, out.emi, out.emf);
    TT_LAUNCH("k_emit_dim0");
    c->launches += 2;
    TT_CUDA(cudaMemcpyAsync(h, tot, 2 * sizeof(u64), cudaMemcpyDeviceToHost, s));
    TT_CUDA(cudaMemcpyAsync(h + 2, mdev, sizeof(u64), cudaMemcpyDeviceToHost, s));
    finish();
}

// The apparent scan of a dense complex goes by vertex pairs, with a word a pair,
// where the threshold keeps at least a kPairShare-th of them. Below, the edges are
// few and short: nearly each needs a scan of its own, a warp has several to do
// one after the other where the next has none, and a warp for each sorted edge is
// faster and takes a word an edge. 12,000 Gaussian points in R^3, whole stage by
// pairs / by edges: 1/64 kept 3.8 / 2.8 ms, 1/8 6.3 / 5.2, 1/4 7.1 / 7.4, 1/2 8.2 / 12;
// 8,000 on a circle 1.85 / 1.24, 3.0 / 2.35, 3.25 / 3.3, 3.9 / 5.5.
constexpr u64 kPairShare = 4;
void dim0(tt_ctx* c, const Complex& cx, u32 maxdim, Dim0Out& out, u64 m_known) {
    out = Dim0Out{};
    if (cx.mat && cx.n >= 2 && cx.n <= kSmallN) {
        dim0_small(c, cx, maxdim, out);
        return;
    }
    u32* err = m_known != kUnknownM ? c->arena.get<u32>(S_DIM0_ERR, 4) : nullptr;
    if (err) TT_CUDA(cudaMemsetAsync(err, 0, sizeof(u32), c->stream));
    const u64 m = sorted_edge_keys(c, cx, 0, !cx.mat && maxdim >= 1, &out.keys, &out.eidx, m_known, err);
    const EdgeFmt fmt{out.eidx};
    out.m = m;
    if (m >= 0xffffffffull) invalid("gb300: more than 2^32 - 1 kept edges");
    const u32 n = cx.n;
    // (packed keys only)
    const bool pairs = cx.mat && n <= kPackedMaxN && m >= u64(n) * (n - (n > 0)) / 2 / kPairShare;
    // per-edge flags
    u8* app = c->arena.get<u8>(S_FLAGS, 2 * m + 16);
    u8* tree = app + m + 8;
    // the apparent scan's results: a word a vertex pair, or arrays by sorted position
    u32* emw = c->arena.get<u32>(S_EDGE_TMP, pairs ? u64(n) * (n - (n > 0)) / 2 + 1 : m + 1);
    u8* emf = pairs ? nullptr : c->arena.get<u8>(S_MISC2, m + 1);
    TT_CUDA(cudaMemsetAsync(tree, 0, m + 1, c->stream));
    // The apparent/emergent scan and the spanning forest read the same sorted
    // edges and write disjoint flags. The forest's short rounds (and their
    // host round trips) run on the side stream, which has the highest
    // priority: its blocks are scheduled ahead of the scan's waiting blocks,
    // and the scan, on the main stream, fills the SMs around them.
    SideScope side(c);
    const cudaStream_t fs = n ? side.fork() : c->stream;   // the forest's stream
    if (maxdim >= 1 && m) {
        const cudaStream_t s = c->stream;
        if (pairs)
            launch_pdl(k_apparent_pairs, dim3(div_up(n, 32), std::min<u32>(div_up(n, 8), 65535)), 256, 0, s, cx.mat, n,
                       cx.thr, emw);
        else if (cx.mat)
            launch_pdl(k_apparent_dense, grid_for(m * 32, 256), 256, 0, s, cx.mat, n, out.keys, fmt, m, app, emw, emf);
        else
            // six of the eight resident blocks an SM: the forest's short
            // kernels then always find free slots instead of waiting for a
            // wave of scan blocks to retire (measured: kNN front end of
            // 100,000 points, dim0 0.04 ms shorter than with all eight)
            launch_pdl(k_apparent_csr, std::min<u32>(grid_for(m, 256), 6 * kSMs), 256, 0, s, 
                CsrCx{cx.rp, cx.ci, cx.w}, out.keys, fmt, c->arena.get<u32>(S_EDGE_INV, m + 1), m, app, emw, emf);
        TT_LAUNCH("k_apparent");
        ++c->launches;
    }
    out.app = maxdim >= 1 ? app : nullptr;
    out.tree = tree;
    // Borůvka spanning forest
    u32* comp = c->arena.get<u32>(S_UF_PARENT, 2 * u64(n) + 2);
    u32* parent = comp + n + 1;
    u32* best = c->arena.get<u32>(S_UF_BEST, n + 1);
    u32* live0 = c->arena.get<u32>(S_UF_WORK, m + 1);
    u32* live1 = c->arena.get<u32>(S_UF_WORK2, m + 1);
    constexpr int kRounds = 64, kPerTrip = 3;
    u32* ctr = c->arena.get<u32>(S_MISC1, 2 * kRounds);   // per round: live count, hooks
    u64 total_hooks = 0;
    if (n) {
        launch_pdl(k_iota, grid_for(n, 256), 256, 0, fs, comp, n);
        launch_pdl(k_iota, grid_for(n, 256), 256, 0, fs, parent, n);
        TT_CUDA(cudaMemsetAsync(best, 0xff, sizeof(u32) * n, fs));
        c->launches += 2;
        TT_CUDA(cudaMemsetAsync(ctr, 0, 2 * kRounds * sizeof(u32), fs));
        // Three rounds a host round trip (a round after convergence finds no
        // edge between components and changes nothing); the grid covers the
        // last live count the host knows (counts only shrink).
        // The edges join in rank order, one group a trip: a component's
        // smallest live edge is its smallest edge of all as soon as any of
        // its edges has joined, so the forest is the same, and the shortest
        // few edges a point connect nearly everything: by the time the long
        // ones join, one pass finds them inside a component (or the forest
        // is complete and they are never read).
        const RankGroups group = rank_groups(m, n);
        u32 known = 0, joined = 0;
        for (int round = 0, trip = 0; round < kRounds; ++trip) {
            const u32 upto = u32(trip < 3 ? group.end[trip] : m);
            if (upto < joined || upto > m) throw Error(TT_ERR_INTERNAL, "gb300: rank groups out of order");
            if (!known && joined == upto) break;
            const int first = round;
            for (int q = 0; q < kPerTrip && round < kRounds; ++q, ++round) {
                launch_pdl(k_bv_offer, grid_for(u64(known) + (upto - joined), 256), 256, 0, fs, out.keys, fmt, live0,
                           round ? ctr + 2 * (round - 1) : nullptr, joined, q ? joined : upto, comp, best, live1,
                           ctr + 2 * round);
                launch_pdl(k_bv_hook, grid_for(n, 256), 256, 0, fs, out.keys, fmt, comp, best, parent, tree, n,
                                                           ctr + 2 * round + 1, ctr + 2 * round);
                launch_pdl(k_bv_flatten, grid_for(n, 256), 256, 0, fs, parent, comp, best, n, ctr + 2 * round);
                TT_LAUNCH("boruvka");
                c->launches += 3;
                std::swap(live0, live1);
            }
            joined = upto;
            u32 h[2 * kPerTrip] = {};
            TT_CUDA(cudaMemcpyAsync(h, ctr + 2 * first, sizeof(u32) * 2 * (round - first), cudaMemcpyDeviceToHost,
                                    fs));
            TT_CUDA(cudaStreamSynchronize(fs));
            const int last = round - first - 1;
            for (int q = 0; q <= last; ++q) total_hooks += h[2 * q + 1];
            known = h[2 * last];
            if (total_hooks == u64(n) - 1) break;                      // one component
            if (h[2 * last + 1] == 0) known = 0;                       // nothing left to merge among the joined
        }
    }
    side.join();   // the forest's tree flags
    // ordered compaction of H0 deaths and columns
    const int want_cols = maxdim >= 1;
    const u64 runs = (m + kRun - 1) / kRun;
    u64* cnt = c->arena.get<u64>(S_MISC0, runs + 1);
    u64* tot = c->arena.get<u64>(S_COUNT, 4);
    const u32 gr = grid_for(runs * 32, 256);
    if (m) {
        if (pairs) launch_pdl(k_count_dim0<true>, gr, 256, 0, c->stream, out.keys, fmt, tree, app, emw, m, static_cast<const u64*>(nullptr), want_cols, cnt);
        else launch_pdl(k_count_dim0<false>, gr, 256, 0, c->stream, out.keys, fmt, tree, app, emw, m, static_cast<const u64*>(nullptr), want_cols, cnt);
        TT_LAUNCH("k_count_dim0");
        scan_exclusive<u64>(c, cnt, cnt, runs, tot);
        c->launches += 1;
    } else {
        TT_CUDA(cudaMemsetAsync(tot, 0, sizeof(u64), c->stream));
    }
    // the outputs: at their largest sizes (H0 bars < n, columns <= m) when
    // that is small, so the emit is enqueued before the counts come back;
    // otherwise at the counted sizes, after the round trip
    auto emit = [&](u64 nh0, u64 ncols) {
        out.h0 = c->arena.get<f32>(S_OUT0, nh0 + 1);
        out.cidx = c->arena.get<u64>(S_OUT1, ncols + 1);
        out.cd = c->arena.get<f32>(S_OUT2, ncols + 1);
        out.emi = c->arena.get<u64>(S_OUT3, ncols + 1);
        out.emf = c->arena.get<u8>(S_OUT4, ncols + 1);
        out.h0_edge = c->arena.get<u64>(S_OUT5, nh0 + 1);
        if (m) {
            auto go = [&](auto kernel) {
                launch_pdl(kernel, gr, 256, 0, c->stream, out.keys, fmt, tree, app, emw, emf, m, static_cast<const u64*>(nullptr), want_cols, cnt, tot,
                           out.h0, out.h0_edge, out.cidx, out.cd, out.emi, out.emf);
            };
            if (pairs) go(k_emit_dim0<true>);
            else go(k_emit_dim0<false>);
            TT_LAUNCH("k_emit_dim0");
            ++c->launches;
        }
    };
    const bool early = m <= (u64(1) << 24);
    if (early) emit(n, want_cols ? m : 0);
    u64 hp = 0;
    u32 bad = 0;
    TT_CUDA(cudaMemcpyAsync(&hp, tot, sizeof(hp), cudaMemcpyDeviceToHost, c->stream));
    if (err) TT_CUDA(cudaMemcpyAsync(&bad, err, sizeof(bad), cudaMemcpyDeviceToHost, c->stream));
    TT_CUDA(cudaStreamSynchronize(c->stream));
    if (bad) throw Error(TT_ERR_INTERNAL, "gb300: more kept edges than announced");
    const u64 h[2] = {hp >> 32, hp & 0xffffffffull};
    out.nh0 = h[0];
    out.ncols = h[1];
    if (!early) emit(h[0], h[1]);
    // every hook merged two components through one tree edge
    out.essential = n - total_hooks;
}

namespace {
__global__ void k_emit_redzed(const u64* __restrict__ keys, EdgeFmt fmt, u64 m, f32* __restrict__ d,
                              int32_t* __restrict__ v) {
    for (u64 e = u64(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += u64(gridDim.x) * blockDim.x) {
        const u64 k = keys[e];
        u32 a, b;
        decode_edge(fmt.redzed(k), a, b);
        d[e] = fmt.d(k);
        v[2 * e] = int32_t(b);
        v[2 * e + 1] = int32_t(a);
    }
}
}  // namespace

// redzed::detail::build_edges (redzed.hpp:545-613): kept edges in
// (d asc, combinatorial index asc) order, vertices (i < j). Writes up to cap
// edges to the device buffers d / verts and returns the edge count.
u64 redzed_edges(tt_ctx* c, const Complex& cx, f32* d, int32_t* verts, u64 cap) {
    u64* keys = nullptr;
    u64* eidx = nullptr;
    const u64 m = sorted_edge_keys(c, cx, 1, false, &keys, &eidx);
    if (m && m <= cap) {
        k_emit_redzed<<<grid_for(m, 256), 256, 0, c->stream>>>(keys, EdgeFmt{eidx}, m, d, verts);
        TT_LAUNCH("k_emit_redzed");
        ++c->launches;
    }
    return m;
}

// The same edge list in context-owned device arrays sized to its count
// (slots S_RZ_D / S_RZ_V), for the host-buffer entry points.
u64 redzed_edges_owned(tt_ctx* c, const Complex& cx, f32** d, int32_t** verts) {
    u64* keys = nullptr;
    u64* eidx = nullptr;
    const u64 m = sorted_edge_keys(c, cx, 1, false, &keys, &eidx);
    *d = c->arena.get<f32>(S_RZ_D, m + 1);
    *verts = c->arena.get<int32_t>(S_RZ_V, 2 * m + 2);
    if (m) {
        k_emit_redzed<<<grid_for(m, 256), 256, 0, c->stream>>>(keys, EdgeFmt{eidx}, m, *d, *verts);
        TT_LAUNCH("k_emit_redzed");
        ++c->launches;
    }
    return m;
}

}  // namespace tt
