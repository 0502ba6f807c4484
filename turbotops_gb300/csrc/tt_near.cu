// tt_near.cu — the spatial order of the ordered searches (tt_near.cuh).
//
// Up to 8 coordinates the points are sorted along a Morton curve: every
// coordinate is mapped through a smooth distribution function of its sample
// mean and deviation (so that Gaussian tails and uniform cubes both spread
// evenly over the cells) and cut into 2^b cells, the b bits of the
// coordinates interleaved: 22 bits in two radix passes (11 in one up to 8,192
// points). Above 8 coordinates a few bits each no longer make compact cells;
// the points are sorted by their nearest pivot instead (tt_knn.cu
// pivot_order). Any order gives the same results; it only decides how many
// tiles a query reads.
#include "tt_near.cuh"

namespace tt {
namespace near {

namespace {

constexpr u32 kCodeDims = 8;
constexpr u32 kSample = 4096;
constexpr int kStatThreads = 256;

// Mean and scale of every coordinate over at most kSample strided points:
// st[k] = mean, st[8 + k] = 1.702 / deviation (the logistic curve with that
// scale follows the normal distribution function within 0.01).
__global__ void __launch_bounds__(kStatThreads) k_near_stats(const f32* __restrict__ x, u32 n, u32 dim,
                                                            f32* __restrict__ st) {
    pdl_wait();
    pdl_trigger();
    __shared__ f32 part[kStatThreads / 32][2];
    const u32 cnt = min(n, kSample), k = blockIdx.x;   // one block a coordinate
    {
        const f32 c0 = x[k];   // sums relative to one point: no cancellation far from the origin
        f32 s = 0.0f, s2 = 0.0f;
        for (u32 i = threadIdx.x; i < cnt; i += kStatThreads) {
            const f32 d = x[(u64(i) * n / cnt) * dim + k] - c0;
            s += d;
            s2 = fmaf(d, d, s2);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if ((threadIdx.x & 31) == 0) {
            part[threadIdx.x >> 5][0] = s;
            part[threadIdx.x >> 5][1] = s2;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            f32 a = 0.0f, b = 0.0f;
            for (int w = 0; w < kStatThreads / 32; ++w) a += part[w][0], b += part[w][1];
            const f32 m = a / f32(cnt), var = b / f32(cnt) - m * m;
            st[k] = c0 + m;
            st[kCodeDims + k] = var > 0.0f ? 1.702f * rsqrtf(var) : 0.0f;
        }
    }
}

// Morton code of every point, `bits` a coordinate (a non-finite coordinate
// lands in some cell: the conversions saturate).
__global__ void k_near_codes(const f32* __restrict__ x, u32 n, u32 dim, u32 bits, const f32* __restrict__ st,
                             u64* __restrict__ key, u32* __restrict__ val) {
    pdl_wait();
    pdl_trigger();
    const f32 cells = f32(1u << bits);
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        u32 q[kCodeDims];
#pragma unroll
        for (u32 k = 0; k < kCodeDims; ++k) {
            q[k] = 0;
            if (k < dim) {
                const f32 z = (x[u64(i) * dim + k] - st[k]) * st[kCodeDims + k];
                const f32 u = cells / (1.0f + __expf(-z));
                q[k] = min(__float2uint_rz(u), (1u << bits) - 1u);
            }
        }
        u32 code = 0;
        for (int b = int(bits) - 1; b >= 0; --b)
#pragma unroll
            for (u32 k = 0; k < kCodeDims; ++k)
                if (k < dim) code = (code << 1) | ((q[k] >> b) & 1u);
        key[i] = code;
        val[i] = i;
    }
}

// Float bits in an order that integer min / max follow (no NaN).
__device__ __forceinline__ u32 ordered(f32 f) {
    const u32 b = __float_as_uint(f);
    return (b >> 31) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ f32 from_ordered(u32 o) { return __uint_as_float((o >> 31) ? o & 0x7fffffffu : ~o); }

// Tile t: its 32 points' coordinates (coordinate-major, zero-padded to dp)
// and ids, and its box (slots past n left out; a NaN leaves the coordinate
// unbounded: linf's maximum drops it, so the point can be near). One warp a
// tile.
__global__ void __launch_bounds__(128) k_near_tiles(const f32* __restrict__ x, u32 n, u32 dim, u32 dp,
                                                    const u32* __restrict__ perm, u32 ntiles, u32 tpad,
                                                    f32* __restrict__ xt, u32* __restrict__ id, f32* __restrict__ box,
                                                    f32* __restrict__ abox) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31, t = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (t >= ntiles) return;
    const u32 p = t * kTile + lane;
    const bool live = p < n;
    const u32 src = live ? perm[p] : 0xffffffffu;
    id[p] = src;
    for (u32 k = 0; k < dp; ++k) {
        const f32 v = live && k < dim ? x[u64(src) * dim + k] : 0.0f;
        xt[(u64(t) * dp + k) * kTile + lane] = v;
        const u32 lo = __reduce_min_sync(0xffffffffu, ordered(!live ? INFINITY : v == v ? v : -INFINITY));
        const u32 hi = __reduce_max_sync(0xffffffffu, ordered(!live ? -INFINITY : v == v ? v : INFINITY));
        if (lane == 0) {
            box[u64(k) * tpad + t] = from_ordered(lo);
            box[u64(dp + k) * tpad + t] = from_ordered(hi);
            if (abox) {
                abox[(u64(t) * 2) * dp + k] = from_ordered(lo);
                abox[(u64(t) * 2 + 1) * dp + k] = from_ordered(hi);
            }
        }
    }
}

// Super tile s: the box of its (up to) 32 tiles' boxes. One warp each.
__global__ void __launch_bounds__(128) k_near_super(const f32* __restrict__ tbox, u32 ntiles, u32 tpad, u32 nsup,
                                                    u32 spad, u32 dp, f32* __restrict__ sbox) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31, s = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (s >= nsup) return;
    const u32 t = s * 32 + lane;
    for (u32 k = 0; k < dp; ++k) {
        const u32 lo = __reduce_min_sync(0xffffffffu, ordered(t < ntiles ? tbox[u64(k) * tpad + t] : INFINITY));
        const u32 hi = __reduce_max_sync(0xffffffffu, ordered(t < ntiles ? tbox[u64(dp + k) * tpad + t] : -INFINITY));
        if (lane == 0) {
            sbox[u64(k) * spad + s] = from_ordered(lo);
            sbox[u64(dp + k) * spad + s] = from_ordered(hi);
        }
    }
}

// ---- separations between blocks ---------------------------------------------
// For blocks A and B of 128 points (4 tiles): with u = u_AB the gradient of
// the distance at D = c_B - c_A (tt_near.cuh, project) and x in B, q in A,
// |x - q|_p |u|_p' >= u . (x - q) >= min over B of u . x - max over A of u . q,
// and u_BA = -u_AB, so with S_AB = min over x in B of u_AB . (x - r) the
// separation is (S_AB + S_BA) / |u|_p' (any common reference r). One block a
// B: its points relative to r in registers, the directions to 32 blocks A at a
// time in shared memory. Rounding: a sum of DP terms errs by less than 2^-16
// of sum |u_k| ext_k, ext the block's largest |x_k - r_k|, which is taken off
// S; |u|_p' is taken 2^-9 up. A non-finite value anywhere ends in a separation
// of 0. FP32 issue bound: 100,000 x 32 (781 blocks, 2.5e9 multiply-adds) 0.24 ms.
__global__ void __launch_bounds__(64) k_near_centres(const f32* __restrict__ abox, u32 ntiles, u32 dp,
                                                     f32* __restrict__ cen) {
    pdl_wait();
    pdl_trigger();
    const u32 b = blockIdx.x, k = threadIdx.x;
    if (k >= dp) return;
    f32 lo = INFINITY, hi = -INFINITY;
    for (u32 t = b * kBlockTiles; t < min(ntiles, (b + 1) * kBlockTiles); ++t) {
        lo = fminf(lo, abox[(u64(t) * 2) * dp + k]);
        hi = fmaxf(hi, abox[(u64(t) * 2 + 1) * dp + k]);
    }
    cen[u64(b) * dp + k] = 0.5f * lo + 0.5f * hi;
}

template <int DP>
__global__ void __launch_bounds__(128) k_near_sep(const f32* __restrict__ xt, const u32* __restrict__ id,
                                                  const f32* __restrict__ cen, u32 ntiles, u32 nblk, int kind, f32 p,
                                                  float2* __restrict__ out) {
    pdl_wait();
    pdl_trigger();
    __shared__ alignas(16) f32 su[32][DP];
    __shared__ f32 ext[DP], part[32][4];
    const u32 B = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const u32 tile = B * kBlockTiles + w;
    const bool live = tile < ntiles && id[tile * kTile + lane] != 0xffffffffu;
    f32 y[DP];
    if (tid < DP) ext[tid] = 0.0f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < DP; ++k) {
        y[k] = live ? __fsub_rn(xt[(u64(tile) * DP + k) * kTile + lane], cen[k]) : 0.0f;   // r: block 0's centre
        const u32 a = __float_as_uint(fabsf(y[k]));   // (a NaN's bits are above every number's)
        const u32 m = __reduce_max_sync(0xffffffffu, a);
        if (lane == 0) atomicMax(reinterpret_cast<u32*>(&ext[k]), m);
    }
    const f32 pd = p / (p - 1.0f);   // (used for Lp only: p > 1)
    for (u32 A0 = blockIdx.y * 32; A0 < nblk; A0 += gridDim.y * 32) {
        __syncthreads();
        for (u32 e = tid; e < 32 * DP; e += 128) {
            const u32 a = e / DP, k = e % DP;
            f32 u = 0.0f;
            if (A0 + a < nblk) {
                const f32 d = cen[u64(B) * DP + k] - cen[u64(A0 + a) * DP + k];
                u = kind == M_L2 ? d
                    : kind == M_L1 ? (d < 0.0f ? -1.0f : d > 0.0f ? 1.0f : 0.0f)
                                   : copysignf(__powf(fabsf(d), p - 1.0f), d);
                if (kind == M_LP && d == 0.0f) u = 0.0f;
            }
            su[a][k] = u;
        }
        __syncthreads();
#pragma unroll 2
        for (u32 a = 0; a < 32; ++a) {
            f32 s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const float4* u4 = reinterpret_cast<const float4*>(su[a]);
#pragma unroll
            for (int k = 0; k < DP / 4; ++k) {
                const float4 u = u4[k];
                s[0] = fmaf(u.x, y[4 * k], s[0]);
                s[1] = fmaf(u.y, y[4 * k + 1], s[1]);
                s[2] = fmaf(u.z, y[4 * k + 2], s[2]);
                s[3] = fmaf(u.w, y[4 * k + 3], s[3]);
            }
            // (a NaN projection counts as -inf: no separation)
            const f32 v = (s[0] + s[1]) + (s[2] + s[3]);
            const u32 m = __reduce_min_sync(0xffffffffu, ordered(!live ? INFINITY : v == v ? v : -INFINITY));
            if (lane == 0) part[a][w] = from_ordered(m);
        }
        __syncthreads();
        if (tid < 32 && A0 + tid < nblk) {
            const f32 s = fminf(fminf(part[tid][0], part[tid][1]), fminf(part[tid][2], part[tid][3]));
            f32 mag = 0.0f, nrm = 0.0f;
            for (int k = 0; k < DP; ++k) {
                const f32 u = fabsf(su[tid][k]);
                mag = fmaf(u, ext[k], mag);
                nrm += kind == M_L2 ? u * u : kind == M_L1 ? 0.0f : __powf(u, pd);
            }
            if (kind == M_L1) nrm = 1.0f;
            else nrm = nrm >= 0x1p-100f ? (kind == M_L2 ? sqrtf(nrm) : __powf(nrm, 1.0f / pd)) : INFINITY;
            out[u64(A0 + tid) * nblk + B] = make_float2(s - 0x1p-16f * mag, nrm * (1.0f + 0x1p-9f));
        }
    }
}

// sep[A][B] from both directions' sums.
__global__ void __launch_bounds__(256) k_near_sep_join(const float2* __restrict__ s, u32 nblk, f32* __restrict__ sep) {
    pdl_wait();
    pdl_trigger();
    const u32 B = blockIdx.x * blockDim.x + threadIdx.x, A = blockIdx.y;
    if (B >= nblk) return;
    const float2 ab = s[u64(A) * nblk + B], ba = s[u64(B) * nblk + A];
    const f32 g = (ab.x + ba.x) * (1.0f - 0x1p-20f) / fmaxf(ab.y, ba.y);
    sep[u64(A) * nblk + B] = A != B && g > 0.0f && g < INFINITY ? g : 0.0f;
}

// A block takes a super tile, a warp a tile of it.
__global__ void __launch_bounds__(1024) k_near_components(const u32* __restrict__ id, u32 ntiles,
                                                          const u32* __restrict__ comp, u32* __restrict__ cpos,
                                                          u32* __restrict__ tcomp, u32* __restrict__ scomp) {
    pdl_wait();
    pdl_trigger();
    __shared__ u32 lo[32], hi[32];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, t = blockIdx.x * 32 + w;
    u32 a = 0xffffffffu, b = 0;   // smallest and largest component of the tile
    if (t < ntiles) {
        const u32 i = id[t * kTile + lane];
        const u32 cc = i != 0xffffffffu ? comp[i] : 0xffffffffu;
        cpos[t * kTile + lane] = cc;
        a = __reduce_min_sync(0xffffffffu, cc);
        b = __reduce_max_sync(0xffffffffu, i != 0xffffffffu ? cc : 0u);
        if (lane == 0) tcomp[t] = a == b ? a : 0xfffffffeu;
    }
    if (lane == 0) lo[w] = a, hi[w] = b;
    __syncthreads();
    if (w == 0) {
        a = __reduce_min_sync(0xffffffffu, lo[lane]);
        b = __reduce_max_sync(0xffffffffu, hi[lane]);
        if (lane == 0) scomp[blockIdx.x] = a == b ? a : 0xfffffffeu;
    }
}

__global__ void __launch_bounds__(256) k_near_queries(const u32* __restrict__ id, u32 ntiles,
                                                      const u32* __restrict__ cpos,
                                                      const unsigned long long* __restrict__ near,
                                                      const u32* __restrict__ kb, const u32* __restrict__ bd, u32 qw,
                                                      u32* __restrict__ qlist, u32* __restrict__ nq) {
    pdl_wait();
    pdl_trigger();
    const u32 lane = threadIdx.x & 31;
    const u32 warps = (gridDim.x * blockDim.x) >> 5;
    for (u32 t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntiles; t += warps) {
        const u32 p = t * kTile + lane, i = id[p];
        const bool ask = i != 0xffffffffu && (!kb || (near[i] == ~0ull && kb[i] <= bd[cpos[p]]));
        const u32 m = __ballot_sync(0xffffffffu, ask);
        if (!m) continue;
        const u32 cnt = __popc(m), room = (cnt + qw - 1) / qw * qw;
        u32 base = 0;
        if (lane == 0) base = atomicAdd(nq, room);
        base = __shfl_sync(0xffffffffu, base, 0);
        const u32 o = __popc(m & ((1u << lane) - 1u));
        if (ask) qlist[base + o] = p;
        if (lane >= cnt && lane < room) qlist[base + lane] = 0xffffffffu;
    }
}

}  // namespace

void near_components(tt_ctx* c, const View& v, const u32* comp, u32* cpos, u32* tcomp, u32* scomp) {
    launch_pdl(k_near_components, v.nsup, 1024, 0, c->stream, v.id, v.ntiles, comp, cpos, tcomp, scomp);
    TT_LAUNCH("k_near_components");
    ++c->launches;
}

void near_queries(tt_ctx* c, const View& v, u32 dim, const u32* cpos, const unsigned long long* near, const u32* kb,
                  const u32* bd, u32* qlist, u32* nq) {
    TT_CUDA(cudaMemsetAsync(nq, 0, sizeof(u32), c->stream));
    launch_pdl(k_near_queries, std::min<u32>(div_up(v.ntiles, 8), 8 * u32(c->sms)), 256, 0, c->stream, v.id, v.ntiles,
               cpos, near, kb, bd, queries_per_warp(padded_dim(dim)), qlist, nq);
    TT_LAUNCH("k_near_queries");
    ++c->launches;
}

// Slots: S_NEAR_SEP (result), S_NEAR_ST.
void near_separations(tt_ctx* c, View& v, u32 dim, int kind, f32 p) {
    const u32 dp = padded_dim(dim);
    v.nblk = div_up(v.ntiles, kBlockTiles);
    if (dp < kProjectDim || kind == M_LINF || v.n < kSepMinPoints || v.nblk > kSepMaxBlocks) return;
    const u64 pairs = u64(v.nblk) * v.nblk;
    f32* cen = c->arena.get<f32>(S_NEAR_ST, std::max<u64>(u64(v.nblk) * dp, 2 * kCodeDims));
    f32* sep = c->arena.get<f32>(S_NEAR_SEP, 3 * pairs + 2);
    float2* s = reinterpret_cast<float2*>(sep + ((pairs + 1) & ~u64(1)));
    launch_pdl(k_near_centres, v.nblk, 64, 0, c->stream, v.abox, v.ntiles, dp, cen);
    TT_LAUNCH("k_near_centres");
    // enough blocks for the chip when there are few Bs
    const dim3 grid(v.nblk, std::min<u32>(div_up(v.nblk, 32), std::max<u32>(1, 2432 / v.nblk)));
    auto go = [&](auto d) {
        launch_pdl(k_near_sep<decltype(d)::value>, grid, 128, 0, c->stream, v.xt, v.id, static_cast<const f32*>(cen),
                   v.ntiles, v.nblk, kind, p, s);
    };
    if (dp == 16) go(std::integral_constant<int, 16>{});
    else if (dp == 32) go(std::integral_constant<int, 32>{});
    else if (dp == 48) go(std::integral_constant<int, 48>{});
    else go(std::integral_constant<int, 64>{});
    TT_LAUNCH("k_near_sep");
    launch_pdl(k_near_sep_join, dim3(div_up(v.nblk, 256), v.nblk), 256, 0, c->stream, static_cast<const float2*>(s),
               v.nblk, sep);
    TT_LAUNCH("k_near_sep_join");
    c->launches += 3;
    v.sep = sep;
}

// The View of the points in the order perm. Slots: S_NEAR_X, S_NEAR_ID,
// S_NEAR_BOX (results).
View near_regroup(tt_ctx* c, const f32* x, u32 n, u32 dim, const u32* perm) {
    View v;
    const u32 dp = padded_dim(dim);
    v.n = n;
    v.ntiles = div_up(n, kTile);
    v.nsup = div_up(v.ntiles, 32);
    v.tpad = v.nsup * 32;
    v.spad = div_up(v.nsup, 32) * 32;
    f32* xt = c->arena.get<f32>(S_NEAR_X, u64(v.ntiles) * dp * kTile);
    u32* id = c->arena.get<u32>(S_NEAR_ID, u64(v.ntiles) * kTile);
    const bool directions = dp >= kProjectDim;
    f32* tbox = c->arena.get<f32>(S_NEAR_BOX, 2 * u64(dp) * (v.tpad + v.spad + (directions ? v.ntiles : 0)));
    f32* sbox = tbox + 2 * u64(dp) * v.tpad;
    f32* abox = directions ? sbox + 2 * u64(dp) * v.spad : nullptr;
    launch_pdl(k_near_tiles, div_up(v.ntiles, 4), 128, 0, c->stream, x, n, dim, dp, perm, v.ntiles, v.tpad, xt, id, tbox,
               abox);
    TT_LAUNCH("k_near_tiles");
    launch_pdl(k_near_super, div_up(v.nsup, 4), 128, 0, c->stream, static_cast<const f32*>(tbox), v.ntiles, v.tpad,
               v.nsup, v.spad, dp, sbox);
    TT_LAUNCH("k_near_super");
    c->launches += 2;
    v.xt = xt;
    v.id = id;
    v.tbox = tbox;
    v.sbox = sbox;
    v.abox = abox;
    return v;
}

// Slots: near_regroup's; S_TC_KEYS, S_TC_VALS, S_NEAR_ST and the radix sort's
// own while it runs.
View near_order(tt_ctx* c, const f32* x, u32 n, u32 dim) {
    if (dim > kCodeDims) return near_regroup(c, x, n, dim, pivot_order(c, x, n, dim));
    u64* key = c->arena.get<u64>(S_TC_KEYS, n);
    u32* val = c->arena.get<u32>(S_TC_VALS, n);
    f32* st = c->arena.get<f32>(S_NEAR_ST, 2 * kCodeDims);
    const u32 bits = std::max<u32>(1, (n <= 8192 ? 11 : 22) / dim);
    launch_pdl(k_near_stats, dim, kStatThreads, 0, c->stream, x, n, dim, st);
    TT_LAUNCH("k_near_stats");
    launch_pdl(k_near_codes, std::min<u32>(div_up(n, 256), 8 * u32(c->sms)), 256, 0, c->stream, x, n, dim, bits, st,
               key, val);
    TT_LAUNCH("k_near_codes");
    c->launches += 2;
    u64* kb = c->arena.get<u64>(S_SORT_A, n);
    u32* vb = c->arena.get<u32>(S_SORT_VA, n);
    return near_regroup(c, x, n, dim, radix_sort<u32>(c, key, val, n, kb, vb, int(bits * dim)) ? vb : val);
}

}  // namespace near
}  // namespace tt
