// tt_batch.cu — the dense front end of many clouds at once, replayed from a
// captured CUDA graph.
//
// Replaces, for every cloud of a batch, the front end the reference runs per
// persistence() call on a full-Rips cloud (turbotops.hpp:230-259 with the
// RedZeD engine that auto picks for H1 on dense input): make_dense
// (rips.hpp:391-416), enclosing_radius (:370-380) and build_edges
// (redzed.hpp:545-613, kept edges in (d asc, combinatorial index asc) order).
//
// The batch is one block-diagonal complex:
//   k_batch_dense   persistent CTAs pull 32 x 64 distance tiles of every cloud
//                   from one work list (uneven clouds balance themselves) and
//                   fold row maxima
//   k_batch_radius  per-cloud minimum of the row maxima
//   k_batch_hist    kept pairs per row, and every cloud's histogram of its kept
//                   distances over bins linear in the distance
//   scan            of the row counts: per-cloud offsets, the total
//   k_batch_bins    bin offsets per cloud; consecutive bins grouped into items
//                   of at most kItemCap edges, or, where one bin holds more
//                   than kBinMax (ties, tight clusters, and clouds of more than
//                   some 4,000 points: 5,018 in any case), the cloud marked
//                   for the radix sort
//   k_batch_part    the kept edges as keys (d bits << 32 | index) into their
//                   items, in no particular order inside an item
//   k_batch_items   each item ordered in shared memory and written out as
//                   EdgeList (diameter, vertex pair)
// A distance is moved twice that way (into its item, and out in order), where
// the four 8-bit passes of a radix sort read it eight times and wrote it four
// (512 clouds, 312 M kept edges: 13.6 ms with the edge lists, now 4.4). The bin
// of a distance is floor(d * bins / radius) in floats: monotone in d, so the
// bins partition the filtration order whatever the rounding.
// The marked clouds go through
//   k_batch_edges   keys cloud << (31 + ib) | d bits << ib | index, compacted
//                   in (cloud, index) order, a segmented stable radix sort on
//                   the distance bits, and k_batch_emit
// whose kernels return at once when no cloud is marked.
// Buffers are sized for the worst case (every pair kept), so no step reads a
// count back to the host and the whole sequence is captured into a CUDA
// graph once and replayed.
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "tt_dense_tile.cuh"
#include "tt_warp_sort.cuh"

namespace tt {

namespace {

// Square distance tiles of T x T on and above each cloud's diagonal, 256
// threads (tt_dense_tile.cuh: each computed once, an off-diagonal tile
// written twice, row maxima folded); T is picked per batch by the autotuner
// below.
constexpr int BT_THREADS = 32 * dtile::kWarps;
struct TileShape {
    int r, c;
};
constexpr TileShape kShapes[] = {{32, 32}, {64, 64}, {96, 96}};
constexpr int kNumShapes = int(sizeof(kShapes) / sizeof(kShapes[0]));

struct Tile {
    u32 cloud, i0, j0;
};

// Persistent CTAs pull tiles of every cloud from one work list (uneven
// clouds balance themselves). DIM > 0: the dimension at compile time; 0: any.
template <int KIND, int T, int DIM>
__global__ void __launch_bounds__(BT_THREADS)
k_batch_dense(const f32* __restrict__ x, const u64* __restrict__ pt_off, const u64* __restrict__ mat_off,
              const u32* __restrict__ sizes, const Tile* __restrict__ tiles, u32 ntiles, u32 dim, f32 p,
              f32* __restrict__ mats, u32* __restrict__ rowmax, u32* __restrict__ next) {
    __shared__ dtile::Smem<T> sm;
    __shared__ u32 tile_id;
    for (;;) {
        if (threadIdx.x == 0) tile_id = atomicAdd(next, 1u);
        __syncthreads();
        const u32 t = tile_id;   // read before sym_tile's first barrier; rewritten after its last
        if (t >= ntiles) break;
        const Tile tl = tiles[t];
        const u64 po = pt_off[tl.cloud];
        dtile::sym_tile<KIND, DIM, false, T>(x + po * dim, sizes[tl.cloud], dim, p, mats + mat_off[tl.cloud],
                                             rowmax + po, tl.i0, tl.j0, sm);
    }
}

// (A cloud's rows are contiguous: a warp whose 32 rows share one cloud takes
// their minimum first and issues one atomic.)
__global__ void k_batch_radius(const u32* __restrict__ rowmax, const u32* __restrict__ row_cloud, u64 rows,
                               u32* __restrict__ radius) {
    const u32 lane = threadIdx.x & 31;
    const u64 stride = u64(gridDim.x) * blockDim.x;
    for (u64 base = u64(blockIdx.x) * blockDim.x + (threadIdx.x & ~31u); base < rows; base += stride) {
        const u64 r = base + lane;   // whole warps iterate together
        const bool ok = r < rows;
        const u32 c = ok ? row_cloud[r] : 0xffffffffu;
        u32 v = ok ? rowmax[r] : 0xffffffffu;
        const u32 c0 = __shfl_sync(0xffffffffu, c, 0);
        if (__all_sync(0xffffffffu, !ok || c == c0)) {
            v = __reduce_min_sync(0xffffffffu, v);
            if (lane == 0) atomicMin(&radius[c0], v);
        } else if (ok) {
            atomicMin(&radius[c], v);
        }
    }
}

// A run of a cloud's rows holding about kChunkPairs pairs.
struct Chunk {
    u32 cloud, row0, row1;
};
constexpr u64 kChunkPairs = 64 * 1024;
constexpr u32 kMaxBins = 8192;
// A run of kPartPairs pairs of a cloud, in index order.
struct Part {
    u32 cloud, first;
};
constexpr int kPartThreads = 512;
constexpr u32 kPartPer = 16;   // pairs a thread
constexpr u32 kPartPairs = kPartThreads * kPartPer;
constexpr size_t kPartSmemMax = 8 * size_t(kPartPairs) + 10 * size_t(kMaxBins);   // keys, items' words, bins' items
constexpr u32 kItemCap = 3840;                 // edges an item orders at once
constexpr u32 kItemStep = 2304;                // an item: the bins that start in one step of this many edges ...
constexpr u32 kBinMax = kItemCap - kItemStep;  // ... and no bin longer than this
constexpr int kItemThreads = 384;
constexpr u32 kSlots = 1920;                   // linear slots an item's keys are placed by
struct Item {
    u32 begin, end;   // edges of the cloud, relative to its first
};

// What the sort stages know of a cloud (device arrays indexed by cloud).
struct CloudTable {
    const u64* pt_off;
    const u64* mat_off;
    const u32* sizes;
    const u32* bin_off;    // first bin; the next cloud's ends them
    const u32* item_off;   // first item slot
};

__device__ __forceinline__ u32 bin_of(f32 d, f32 scale, u32 bins) {
    return min(bins - 1u, __float2uint_rz(__fmul_rn(d, scale)));   // (a NaN product, 0 * inf, is bin 0)
}

// The kept entries of a row (j < i, d <= thr), a warp a row: f(d, j) for each,
// with kRowLoads loads in flight (a row's entries are used once, so the loads'
// latency is what a warp waits for).
constexpr int kRowLoads = 8;
template <typename F>
__device__ __forceinline__ void for_row(const f32* __restrict__ row, u32 i, f32 thr, F&& f) {
    const u32 lane = threadIdx.x & 31;
    for (u32 j0 = 0; j0 < i; j0 += 32 * kRowLoads) {
        f32 d[kRowLoads];
#pragma unroll
        for (int q = 0; q < kRowLoads; ++q) {
            const u32 j = j0 + 32 * q + lane;
            d[q] = j < i ? row[j] : INFINITY;
        }
        f(d, j0 + lane);
    }
}

// Row counts and the cloud's histogram, one block a chunk: the bins counted in
// shared memory first (one global atomic a bin and chunk).
constexpr int kHistThreads = 512;
__global__ void __launch_bounds__(kHistThreads)
    k_batch_hist(const f32* __restrict__ mats, CloudTable T, const Chunk* __restrict__ chunks,
                 const u32* __restrict__ radius, u64* __restrict__ row_cnt, u32* __restrict__ hist) {
    __shared__ u32 h[kMaxBins];
    const Chunk ck = chunks[blockIdx.x];
    const u32 c = ck.cloud, n = T.sizes[c], b0 = T.bin_off[c], bins = T.bin_off[c + 1] - b0;
    const f32 thr = __uint_as_float(radius[c]), scale = __fdiv_rn(f32(bins), thr);
    for (u32 b = threadIdx.x; b < bins; b += kHistThreads) h[b] = 0;
    __syncthreads();
    const u32 lane = threadIdx.x & 31;
    auto count = [&](auto binned) {
        for (u32 i = ck.row0 + (threadIdx.x >> 5); i < ck.row1; i += kHistThreads / 32) {
            u32 kept = 0;
            for_row(mats + T.mat_off[c] + u64(i) * n, i, thr, [&](const f32(&d)[kRowLoads], u32 j) {
#pragma unroll
                for (int q = 0; q < kRowLoads; ++q) {
                    const bool keep = j + 32 * q < i && d[q] <= thr;
                    if (decltype(binned)::value && keep) atomicAdd(&h[bin_of(d[q], scale, bins)], 1u);
                    kept += keep;
                }
            });
            kept = __reduce_add_sync(0xffffffffu, kept);
            if (lane == 0) row_cnt[T.pt_off[c] + i] = kept;
        }
    };
    if (bins == 1) {   // (a cloud without items)
        count(std::false_type{});
        return;
    }
    count(std::true_type{});
    __syncthreads();
    for (u32 b = threadIdx.x; b < bins; b += kHistThreads)
        if (h[b]) atomicAdd(&hist[b0 + b], h[b]);
}

// Exclusive scan over the 1,024 threads of the block (u32).
__device__ __forceinline__ u32 block_scan1024(u32 v, u32* warp_tot, u32& total) {
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    u32 inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= u32(o)) inc += y;
    }
    __syncthreads();   // warp_tot free again
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    u32 pre = 0, tot = 0;
#pragma unroll
    for (u32 q = 0; q < 32; ++q) {
        const u32 t = warp_tot[q];
        pre += q < w ? t : 0u;
        tot += t;
    }
    total = tot;
    return pre + inc - v;
}

// One block a cloud: its items with the partition's cursors, the item of every
// bin, and whether the cloud is left to the radix sort; edge_off from the
// scanned row counts (the last block adds the total).
__global__ void __launch_bounds__(1024) k_batch_bins(CloudTable T, u32 clouds, const u64* __restrict__ row_off,
                                                     const unsigned long long* __restrict__ total,
                                                     const u32* __restrict__ hist, u16* __restrict__ bin_item,
                                                     Item* __restrict__ items, u32* __restrict__ cursor,
                                                     u32* __restrict__ radix, u64* __restrict__ edge_off) {
    __shared__ u32 wt[32];
    const u32 c = blockIdx.x, b0 = T.bin_off[c], bins = T.bin_off[c + 1] - b0;
    const u32 per = (bins + 1023) / 1024;   // bins a thread: at most kMaxBins / 1024
    u32 v[kMaxBins / 1024];
    u32 sum = 0, mx = 0;
#pragma unroll
    for (u32 q = 0; q < kMaxBins / 1024; ++q) {
        const u32 b = threadIdx.x * per + q;
        v[q] = q < per && b < bins ? hist[b0 + b] : 0u;
        sum += v[q];
        mx = max(mx, v[q]);
    }
    u32 all;
    const u32 start = block_scan1024(sum, wt, all);
    const u32 s0 = T.item_off[c], cap = T.item_off[c + 1] - s0;
    const bool rad = __syncthreads_or(mx > kBinMax) || cap == 0;
    if (threadIdx.x == 0) {
        radix[c] = rad;
        edge_off[c] = row_off[T.pt_off[c]];
        if (c == clouds - 1) edge_off[clouds] = *total;
    }
    // items: bin b opens one when its start lies in another step than the
    // start of the bin before it
    u32 opens = 0, run = start;
    u32 prev = threadIdx.x == 0 ? 0xffffffffu : 0u;   // the previous bin's step
    // the previous bin (another thread's last) starts at start - its count; its step:
    __shared__ u32 last_step[1024];
#pragma unroll
    for (u32 q = 0, r = start; q < kMaxBins / 1024; ++q) {
        if (q < per) last_step[threadIdx.x] = r / kItemStep;
        r += v[q];
    }
    __syncthreads();
    if (threadIdx.x > 0) prev = last_step[threadIdx.x - 1];
#pragma unroll
    for (u32 q = 0, r = start, p = prev; q < kMaxBins / 1024; ++q) {
        const u32 b = threadIdx.x * per + q;
        if (q < per && b < bins) {
            const u32 st = r / kItemStep;
            opens += st != p;
            p = st;
        }
        r += v[q];
    }
    u32 nitems;
    u32 slot = block_scan1024(opens, wt, nitems);
    u32 p = prev;
#pragma unroll
    for (u32 q = 0; q < kMaxBins / 1024; ++q) {
        const u32 b = threadIdx.x * per + q;
        if (q < per && b < bins) {
            const u32 st = run / kItemStep;
            if (st != p && !rad) {
                items[s0 + slot].begin = run;
                cursor[s0 + slot] = run;
                if (slot) items[s0 + slot - 1].end = run;
            }
            slot += st != p;
            p = st;
            bin_item[b0 + b] = u16(slot - 1);
        }
        run += v[q];
    }
    if (rad) nitems = 0;
    else if (threadIdx.x == 0 && nitems) items[s0 + nitems - 1].end = all;
    for (u32 q = nitems + threadIdx.x; q < cap; q += blockDim.x) items[s0 + q] = Item{0, 0};
}

// decode_edge for idx < 2^31 in 32-bit arithmetic (v <= 65,536, so v (v - 1)
// fits; the closed form in FP32 is within one of the answer, whose 2^17 steps
// are far wider than the approximate root's relative error of 2^-22).
__device__ __forceinline__ void decode_edge31(u32 idx, u32& a, u32& b) {
    f32 r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(fmaf(8.0f, f32(idx), 1.0f)));
    u32 v = u32((1.0f + r) * 0.5f);
    u32 t = v * (v - 1u) / 2u;
    if (t > idx) {
        --v;
        t -= v;
    }
    if (t + v <= idx) {
        t += v;
        ++v;
    }
    a = v;
    b = idx - t;
}

// The kept edges of a run of pairs into their items, one block a run: counted
// by item, placed item by item in shared memory and written from there, so
// that the stores of a warp are runs of neighbouring words (1,100 points: 240
// items, 25 edges a run); the places in an item come from its cursor. Written
// directly into 8,192 bins, every edge's store was a sector of its own: 3.45 ms
// for 312 M edges, now 1.79 (6,144 pairs a block 2.4, 12,288 2.6).
__global__ void __launch_bounds__(kPartThreads, 2)
    k_batch_part(const f32* __restrict__ mats, CloudTable T, const Part* __restrict__ parts,
                 const u32* __restrict__ radius, const u32* __restrict__ radix, const u64* __restrict__ edge_off,
                 const u16* __restrict__ bin_item, u32* __restrict__ cursor, u32 max_items, u64* __restrict__ keys) {
    extern __shared__ u64 sk[];   // [kPartPairs]
    u32* cnt = reinterpret_cast<u32*>(sk + kPartPairs);   // [max_items] edges, then the first place
    u32* to = cnt + max_items;                            // [max_items] the item's place in the keys less cnt
    u16* item_of = reinterpret_cast<u16*>(to + max_items);   // [bins]
    __shared__ u32 wt[kPartThreads / 32];
    const Part pt = parts[blockIdx.x];
    const u32 c = pt.cloud;
    if (radix[c]) return;
    const u32 n = T.sizes[c], b0 = T.bin_off[c], bins = T.bin_off[c + 1] - b0;
    const u32 s0 = T.item_off[c], items = min(T.item_off[c + 1] - s0, bins);
    const u32 pairs = u32(u64(n) * (n - 1) / 2), m = min(kPartPairs, pairs - pt.first);
    const f32 thr = __uint_as_float(radius[c]), scale = __fdiv_rn(f32(bins), thr);
    const u32 tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const f32* mat = mats + T.mat_off[c];
    f32 d[kPartPer];
#pragma unroll
    for (u32 q = 0; q < kPartPer; ++q) {
        const u32 e = q * kPartThreads + tid;
        u32 i, j;
        decode_edge31(pt.first + e, i, j);
        d[q] = e < m ? mat[u64(i) * n + j] : INFINITY;
    }
    for (u32 b = tid; b < items; b += kPartThreads) cnt[b] = 0;
    for (u32 b = tid; b < bins; b += kPartThreads) item_of[b] = bin_item[b0 + b];
    __syncthreads();
    u32 at[kPartPer];   // item, place in it (both below 2^13)
#pragma unroll
    for (u32 q = 0; q < kPartPer; ++q) {
        const u32 e = q * kPartThreads + tid;
        at[q] = 0xffffffffu;
        if (e < m && d[q] <= thr) {
            const u32 it = item_of[bin_of(d[q], scale, bins)];
            at[q] = it << 16 | atomicAdd(&cnt[it], 1u);
        }
    }
    __syncthreads();
    const u32 per = (items + kPartThreads - 1) / kPartThreads, b1 = min(items, (tid + 1) * per);
    u32 sum = 0;
    for (u32 b = tid * per; b < b1; ++b) sum += cnt[b];
    u32 inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= u32(o)) inc += y;
    }
    if (lane == 31) wt[w] = inc;
    __syncthreads();
    u32 run = inc - sum, kept = 0;
#pragma unroll
    for (u32 q = 0; q < kPartThreads / 32; ++q) {
        run += q < w ? wt[q] : 0u;
        kept += wt[q];
    }
    for (u32 b = tid * per; b < b1; ++b) {
        const u32 k = cnt[b];
        cnt[b] = run;
        to[b] = (k ? atomicAdd(&cursor[s0 + b], k) : 0u) - run;
        run += k;
    }
    __syncthreads();
#pragma unroll
    for (u32 q = 0; q < kPartPer; ++q)
        if (at[q] != 0xffffffffu)
            sk[cnt[at[q] >> 16] + (at[q] & 0xffffu)] =
                (u64(__float_as_uint(d[q])) << 32) | (pt.first + q * kPartThreads + tid);
    __syncthreads();
    u64* out = keys + edge_off[c];
    for (u32 e = tid; e < kept; e += kPartThreads) {
        const u64 key = sk[e];
        out[to[item_of[bin_of(__uint_as_float(u32(key >> 32)), scale, bins)]] + e] = key;
    }
}

// One item: its keys counted into kSlots linear slots of its distance range
// (about one key a slot), placed slot by slot in shared memory, and the few
// keys of a slot put in order by insertion (order_crowded where distances crowd:
// a slot of more than kSlotMax keys). Then written out in order. Bound by shared-memory latency and so by the warps
// an SM: 312 M edges 3.1 ms with 256 threads on up to 4,096 keys (23 warps an
// SM), now 2.17 with 384 on up to 3,840 (40 registers, 48 warps).
constexpr u32 kSlotMax = 24;
constexpr u32 kSlotWarp = 512;

// A few keys in order, by insertion of the whole key.
__device__ __forceinline__ void order_few(u64* k, u32 len) {
    for (u32 x = 1; x < len; ++x) {
        const u64 key = k[x];
        u32 y = x;
        while (y > 0 && k[y - 1] > key) {
            k[y] = k[y - 1];
            --y;
        }
        k[y] = key;
    }
}

template <int K>
__device__ __forceinline__ void order_ties(u64* __restrict__ k, u32 len, u32 d) {
    const u32 lane = threadIdx.x & 31;
    u32 idx[K];
#pragma unroll
    for (u32 q = 0; q < K; ++q) idx[q] = q * 32 + lane < len ? u32(k[q * 32 + lane]) : 0xffffffffu;
    sort_lane_keys<K>(idx);
    __syncwarp();
#pragma unroll
    for (u32 q = 0; q < K; ++q)
        if (lane * K + q < len) k[lane * K + q] = (u64(d) << 32) | idx[q];
}

// A crowded slot's keys (at most kSlotWarp) in order, by one warp: ties by
// their indices in registers, else an odd-even transposition.
__device__ __forceinline__ void order_crowd(u64* k, u32 len) {
    const u32 lane = threadIdx.x & 31, d = u32(k[0] >> 32);
    bool ties = true;
    for (u32 e = lane; e < len; e += 32) ties = ties && u32(k[e] >> 32) == d;
    if (__all_sync(0xffffffffu, ties)) {
        if (len <= 64) order_ties<2>(k, len, d);
        else if (len <= 128) order_ties<4>(k, len, d);
        else if (len <= 256) order_ties<8>(k, len, d);
        else order_ties<kSlotWarp / 32>(k, len, d);
        return;
    }
    for (u32 p = 0; p < len; ++p) {
        for (u32 e = (p & 1u) + 2 * lane; e + 1 < len; e += 64) {
            const u64 x = k[e], y = k[e + 1];
            if (x > y) {
                k[e] = y;
                k[e + 1] = x;
            }
        }
        __syncwarp();
    }
}

// A placed item (first[s]: the first of slot s's keys, m in all) with crowded
// slots: a warp orders such a slot; where one holds more than kSlotWarp keys, the
// block the whole item by a bitonic sort. (64 clouds of 300 lattice points, slots
// of up to 300 ties: 189 us with the bitonic sort for every such item, 49 so. A
// function of its own: beside the common case its code cost that 1 to 3 %.)
__device__ __noinline__ void order_crowded(u64* sk, const u32* first, u32 m) {
    __shared__ u16 crowd[kItemCap / (kSlotMax + 1) + 1];   // the crowded slots
    __shared__ u32 ncrowd;
    const u32 tid = threadIdx.x;
    auto len_of = [&](u32 s) -> u32 { return (s + 1 < kSlots ? first[s + 1] : m) - first[s]; };
    if (tid == 0) ncrowd = 0;
    __syncthreads();
    u32 most = 0;
    for (u32 s = tid; s < kSlots; s += kItemThreads) {
        const u32 len = len_of(s);
        if (len > kSlotMax) crowd[atomicAdd(&ncrowd, 1u)] = u16(s);
        most = max(most, len);
    }
    if (!__syncthreads_or(most > kSlotWarp)) {
        for (u32 s = tid; s < kSlots; s += kItemThreads) {
            const u32 len = len_of(s);
            if (len <= kSlotMax) order_few(sk + first[s], len);
        }
        for (u32 q = tid >> 5; q < ncrowd; q += kItemThreads / 32) order_crowd(sk + first[crowd[q]], len_of(crowd[q]));
        return;
    }
    u32 P = 2;
    while (P < m) P <<= 1;
    for (u32 e = m + tid; e < P; e += kItemThreads) sk[e] = ~0ull;
    __syncthreads();
    for (u32 size = 2; size <= P; size <<= 1)
        for (u32 stride = size >> 1; stride; stride >>= 1) {
            for (u32 i = tid; i < P / 2; i += kItemThreads) {
                const u32 a = 2 * i - (i & (stride - 1)), b = a + stride;
                const u64 x = sk[a], y = sk[b];
                if ((x > y) == ((a & size) == 0)) {
                    sk[a] = y;
                    sk[b] = x;
                }
            }
            __syncthreads();
        }
}

__global__ void __launch_bounds__(kItemThreads, 4)
    k_batch_items(const Item* __restrict__ items, const u32* __restrict__ item_cloud, const u64* __restrict__ edge_off,
                  const u64* __restrict__ keys, f32* __restrict__ ed, int32_t* __restrict__ ev) {
    __shared__ u64 sk[4096];   // kItemCap, up to the bitonic sort's power of two
    __shared__ u32 cnt[kSlots];
    __shared__ u32 red[2][kItemThreads / 32];
    __shared__ u32 wt[kItemThreads / 32];
    const Item it = items[blockIdx.x];
    const u32 m = it.end - it.begin;
    if (m == 0) return;
    const u64 base = edge_off[item_cloud[blockIdx.x]] + it.begin;
    const u32 tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    constexpr u32 kPer = kItemCap / kItemThreads;
    static_assert(kPer * kItemThreads == kItemCap && kSlots % kItemThreads == 0 && kSlots <= kItemCap && kItemCap <= 4096);
    u64 k[kPer];
    u32 lo = 0xffffffffu, hi = 0;
#pragma unroll
    for (u32 q = 0; q < kPer; ++q) {
        const u32 e = q * kItemThreads + tid;
        if (e < kSlots) cnt[e] = 0;
        k[q] = e < m ? keys[base + e] : ~0ull;
        if (e < m) {
            lo = min(lo, u32(k[q] >> 32));
            hi = max(hi, u32(k[q] >> 32));
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) red[0][w] = lo, red[1][w] = hi;
    __syncthreads();
#pragma unroll
    for (u32 q = 0; q < kItemThreads / 32; ++q) lo = min(lo, red[0][q]), hi = max(hi, red[1][q]);
    // slots linear in the distance: (d - dmin) * (kSlots / (dmax - dmin)), monotone in d
    const f32 dmin = __uint_as_float(lo), range = __fsub_rn(__uint_as_float(hi), dmin);
    const f32 scale = range > 0.0f ? __fdiv_rn(f32(kSlots), range) : 0.0f;
    u32 at[kPer];
#pragma unroll
    for (u32 q = 0; q < kPer; ++q) {
        const u32 e = q * kItemThreads + tid;
        if (q * kItemThreads >= m) break;
        if (e < m) {
            const f32 d = __uint_as_float(u32(k[q] >> 32));
            const u32 s = bin_of(__fsub_rn(d, dmin), scale, kSlots);
            at[q] = (s << 16) | atomicAdd(&cnt[s], 1u);   // slot, place in it (both below 2^13)
        }
    }
    __syncthreads();
    // exclusive scan of the slots, kSlotPer consecutive ones a thread
    constexpr u32 kSlotPer = kSlots / kItemThreads;
    u32 c[kSlotPer], sum = 0, most = 0;
#pragma unroll
    for (u32 q = 0; q < kSlotPer; ++q) {
        c[q] = cnt[tid * kSlotPer + q];
        sum += c[q];
        most = max(most, c[q]);
    }
    u32 inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= u32(o)) inc += y;
    }
    if (lane == 31) wt[w] = inc;
    const bool crowded = __syncthreads_or(most > kSlotMax);
    u32 pre = inc - sum;
#pragma unroll
    for (u32 q = 0; q < kItemThreads / 32; ++q) pre += q < w ? wt[q] : 0u;
    {
        u32 run = pre;
#pragma unroll
        for (u32 q = 0; q < kSlotPer; ++q) {
            cnt[tid * kSlotPer + q] = run;
            run += c[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (u32 q = 0; q < kPer; ++q) {
        const u32 e = q * kItemThreads + tid;
        if (q * kItemThreads >= m) break;
        if (e < m) sk[cnt[at[q] >> 16] + (at[q] & 0xffffu)] = k[q];
    }
    __syncthreads();
    if (!crowded) {
        u32 run = pre;
#pragma unroll
        for (u32 q = 0; q < kSlotPer; ++q) {
            order_few(sk + run, c[q]);
            run += c[q];
        }
    } else {
        order_crowded(sk, cnt, m);
    }
    __syncthreads();
    for (u32 e = tid; e < m; e += kItemThreads) {
        const u64 key = sk[e];
        u32 a, b;
        decode_edge31(u32(key), a, b);
        ed[base + e] = __uint_as_float(u32(key >> 32));
        reinterpret_cast<int2*>(ev)[base + e] = make_int2(int(b), int(a));
    }
}

// The marked clouds' kept pairs written compacted, at row_off[row] + rank in
// the row: their keys run over (cloud, index) ascending (rows ascending, j
// ascending in a row), so a stable sort on the bits above the index field
// alone orders them by (cloud, d, index). Key: cloud << (31 + ib) | d bits << ib | index.
__global__ void k_batch_edges(const f32* __restrict__ mats, const u64* __restrict__ mat_off,
                              const u32* __restrict__ sizes, const u64* __restrict__ pt_off,
                              const u32* __restrict__ row_cloud, u64 rows, const u32* __restrict__ radius,
                              const u32* __restrict__ radix, int ib, const u64* __restrict__ row_off,
                              u64* __restrict__ keys) {
    const int lane = threadIdx.x & 31;
    const u64 warps = (u64(gridDim.x) * blockDim.x) >> 5;
    for (u64 r = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
        const u32 c = row_cloud[r];
        if (!radix[c]) continue;
        const u32 n = sizes[c];
        const u32 i = u32(r - pt_off[c]);
        const f32 thr = __uint_as_float(radius[c]);
        const f32* row = mats + mat_off[c] + u64(i) * n;
        const u64 rbase = u64(i) * (i - 1) / 2;
        u64 pos = row_off[r];
#pragma unroll 4
        for (u32 j0 = 0; j0 < i; j0 += 32) {
            const u32 j = j0 + lane;
            const f32 d = j < i ? row[j] : INFINITY;
            const bool keep = j < i && d <= thr;
            const u32 bal = __ballot_sync(0xffffffffu, keep);
            if (keep)
                keys[pos + __popc(bal & ((1u << lane) - 1u))] =
                    (u64(c) << (31 + ib)) | (u64(__float_as_uint(d)) << ib) | (rbase + j);
            pos += __popc(bal);
        }
    }
}

// The segmented sort's tiles of the marked clouds' keys: cloud c's
// ceil(count / kSegTileKeys) tiles after the previous ones', their digit
// counts at 256 per tile in the same order; *ntiles = the list's length. One
// block; clouds <= 65536. place[c]: the cloud's first tile and the keys before
// it; a group of threads a cloud then writes its tiles (by one thread a cloud,
// 48,800 tiles of 20,000 points took 779 us).
__global__ void __launch_bounds__(1024) k_batch_tiles(const u64* __restrict__ off, const u32* __restrict__ radix,
                                                      u32 clouds, uint2* __restrict__ place,
                                                      SegTile* __restrict__ tiles, u32* __restrict__ ntiles) {
    __shared__ u32 wt[32];
    const u32 t = threadIdx.x, per = (clouds + blockDim.x - 1) / blockDim.x;
    auto keys_of = [&](u32 c) -> u32 { return radix[c] ? u32(off[c + 1] - off[c]) : 0u; };
    u32 sum = 0, ksum = 0;
    for (u32 c = t * per; c < min(clouds, (t + 1) * per); ++c) {
        sum += (keys_of(c) + kSegTileKeys - 1) / kSegTileKeys;
        ksum += keys_of(c);
    }
    u32 total, ktotal;
    u32 run = block_scan1024(sum, wt, total), krun = block_scan1024(ksum, wt, ktotal);
    if (t == 0) *ntiles = total;
    if (total == 0) return;
    for (u32 c = t * per; c < min(clouds, (t + 1) * per); ++c) {
        place[c] = make_uint2(run, krun);
        run += (keys_of(c) + kSegTileKeys - 1) / kSegTileKeys;
        krun += keys_of(c);
    }
    __syncthreads();
    u32 group = 32;   // threads a cloud
    while (group < 1024 && u64(clouds) * group * 2 <= 1024) group *= 2;
    for (u32 c = t / group; c < clouds; c += 1024 / group) {
        const u32 tc = (keys_of(c) + kSegTileKeys - 1) / kSegTileKeys;
        if (!tc) continue;
        const uint2 at = place[c];
        for (u32 q = t % group; q < tc; q += group)
            tiles[at.x + q] = SegTile{c, q, 256u * at.x, tc, u32(off[c]) - at.y};
    }
}

__global__ void k_batch_emit(const u64* __restrict__ keys, const u64* __restrict__ off,
                             const SegTile* __restrict__ tiles, const u32* __restrict__ ntiles, int ib,
                             f32* __restrict__ d, int32_t* __restrict__ verts) {
    const u64 imask = (1ull << ib) - 1;
    const u32 nt = *ntiles;
    for (u32 q = blockIdx.x; q < nt; q += gridDim.x) {
        const SegTile tl = tiles[q];
        const u64 lo = off[tl.seg] + u64(tl.t) * kSegTileKeys, hi = min(lo + kSegTileKeys, off[tl.seg + 1]);
        for (u64 e = lo + threadIdx.x; e < hi; e += blockDim.x) {
            const u64 k = keys[e];
            u32 a, b;
            decode_edge(k & imask, a, b);
            d[e] = __uint_as_float(u32((k >> ib) & 0x7fffffffu));
            verts[2 * e] = int32_t(b);
            verts[2 * e + 1] = int32_t(a);
        }
    }
}

}  // namespace

struct Batch {
    tt_ctx* owner = nullptr;
    tt_ctx sctx;   // capture stream + own arena for the sort's scratch
    u32 clouds = 0, dim = 0, maxn = 0;
    int kind = 0;
    f32 p = 2.0f;
    int ib = 0;
    u64 total_pts = 0, total_mat = 0, total_pairs = 0;
    // device buffers (one cudaMalloc each, owned)
    f32* x = nullptr;
    f32* mats = nullptr;
    u32* rowmax = nullptr;
    u32* radius = nullptr;
    u64* pt_off = nullptr;
    u64* mat_off = nullptr;
    u32* sizes = nullptr;
    Tile* tiles[kNumShapes] = {};
    u32 ntiles[kNumShapes] = {};
    int shape = 1;                      // index into kShapes
    bool tuned = false, tuned_from_cache = false;
    float tune_ms[kNumShapes] = {};
    u32* row_cloud = nullptr;
    u32* next = nullptr;
    u64* keys = nullptr;
    u64* kbuf = nullptr;       // the sort's other buffer
    u64* row_cnt = nullptr;    // kept pairs per row, then their exclusive scan
    u64* row_off = nullptr;
    unsigned long long* count = nullptr;
    Chunk* chunks = nullptr;        // row runs of the histogram
    u32 nchunks = 0;
    Part* parts = nullptr;          // pair runs of the partition
    u32 nparts = 0;
    u32 part_items = 0;             // most items of a cloud
    size_t part_smem = 0;
    u32* bin_off = nullptr;         // first bin of every cloud
    u32 total_bins = 0;
    u32* hist = nullptr;            // bin counts
    u16* bin_item = nullptr;        // the item of every bin
    u32* item_off = nullptr;        // first item slot of every cloud
    u32 total_items = 0;
    Item* items = nullptr;
    u32* cursor = nullptr;          // the next free place of every item
    u32* item_cloud = nullptr;
    u32* radix = nullptr;           // clouds left to the radix sort
    u64* edge_off = nullptr;
    uint2* tile_place = nullptr;    // a marked cloud's first tile, the keys before it
    SegTile* seg_tiles = nullptr;   // the segmented sort's tiles of the kept keys (built on the device)
    u32* seg_ntiles = nullptr;      // ... their number
    u32 nseg_tiles = 0;             // capacity: every cloud's largest key count in tiles
    u32 sure_tiles = 0;             // ... of the clouds that have no items
    u64 seg_hist = 0;               // the digit counts' capacity: 256 per tile
    f32* ed = nullptr;
    int32_t* ev = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    u64 graph_kernels = 0;   // kernels one run launches
    bool use_graph = true;
    std::vector<void*> owned;

    template <typename T>
    T* alloc(u64 count) {
        void* p = nullptr;
        const cudaError_t e = cudaMalloc(&p, std::max<u64>(count, 1) * sizeof(T));
        if (e != cudaSuccess) {
            cudaGetLastError();
            throw Error(TT_ERR_LENGTH, "gb300: batch buffers exceed device memory");
        }
        owned.push_back(p);
        return static_cast<T*>(p);
    }

    template <int T, int D>
    void launch_dense_kd(u32 grid, u32 nt, const Tile* tl, cudaStream_t s) {
        switch (kind) {
            case M_L1: k_batch_dense<M_L1, T, D><<<grid, BT_THREADS, 0, s>>>(x, pt_off, mat_off, sizes, tl, nt, dim, p, mats, rowmax, next); break;
            case M_L2: k_batch_dense<M_L2, T, D><<<grid, BT_THREADS, 0, s>>>(x, pt_off, mat_off, sizes, tl, nt, dim, p, mats, rowmax, next); break;
            case M_LINF: k_batch_dense<M_LINF, T, D><<<grid, BT_THREADS, 0, s>>>(x, pt_off, mat_off, sizes, tl, nt, dim, p, mats, rowmax, next); break;
            default: k_batch_dense<M_LP, T, D><<<grid, BT_THREADS, 0, s>>>(x, pt_off, mat_off, sizes, tl, nt, dim, p, mats, rowmax, next); break;
        }
    }
    template <int T>
    void launch_dense_t(int si, cudaStream_t s) {
        const u32 nt = ntiles[si];
        const u32 grid = u32(std::max<u64>(1, std::min<u64>(nt, u64(owner->sms) * 8)));
        const Tile* tl = tiles[si];
        if (dim == 3) launch_dense_kd<T, 3>(grid, nt, tl, s);
        else launch_dense_kd<T, 0>(grid, nt, tl, s);
        TT_LAUNCH("k_batch_dense");
    }
    void launch_dense(int si, cudaStream_t s) {
        switch (si) {
            case 0: launch_dense_t<32>(si, s); break;
            case 1: launch_dense_t<64>(si, s); break;
            default: launch_dense_t<96>(si, s); break;
        }
    }

    // The autotuner: every tile shape times the distance pass once on this
    // batch (CUDA events on the batch's stream, after one untimed pass that
    // loads the kernels); the fastest serves every later run. The pick is
    // cached per (metric, dimension, cloud count, size classes), so later
    // batches of the same kind skip the timing.
    void tune() {
        static std::mutex mu;
        static std::map<std::string, int> cache;
        std::string key = std::to_string(kind) + "/" + std::to_string(dim) + "/" + std::to_string(clouds) + "/" +
                          std::to_string(maxn >> 6) + "/" + std::to_string(total_pts >> 12);
        {
            std::lock_guard<std::mutex> l(mu);
            auto it = cache.find(key);
            if (it != cache.end()) {
                shape = it->second;
                tuned_from_cache = true;
                return;
            }
        }
        cudaStream_t s = sctx.stream;
        cudaEvent_t e0, e1;
        TT_CUDA(cudaEventCreate(&e0));
        TT_CUDA(cudaEventCreate(&e1));
        float best = 0;
        int pick = 1;
        for (int si = 0; si < kNumShapes; ++si) {
            for (int rep = 0; rep < 2; ++rep) {
                TT_CUDA(cudaMemsetAsync(rowmax, 0, total_pts * sizeof(u32), s));
                TT_CUDA(cudaMemsetAsync(next, 0, sizeof(u32), s));
                TT_CUDA(cudaEventRecord(e0, s));
                launch_dense(si, s);
                TT_CUDA(cudaEventRecord(e1, s));
                sctx.launches += 1;
            }
            TT_CUDA(cudaEventSynchronize(e1));
            float ms = 0;
            TT_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            tune_ms[si] = ms;
            if (si == 0 || ms < best) {
                best = ms;
                pick = si;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        shape = pick;
        std::lock_guard<std::mutex> l(mu);
        cache[key] = pick;
    }

    void enqueue() {
        cudaStream_t s = sctx.stream;
        TT_CUDA(cudaMemsetAsync(rowmax, 0, total_pts * sizeof(u32), s));
        TT_CUDA(cudaMemsetAsync(radius, 0xff, clouds * sizeof(u32), s));
        TT_CUDA(cudaMemsetAsync(next, 0, sizeof(u32), s));
        TT_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long), s));
        TT_CUDA(cudaMemsetAsync(hist, 0, total_bins * sizeof(u32), s));
        launch_dense(shape, s);

        const u32 g2 = u32(std::min<u64>((total_pts + 255) / 256, u64(owner->sms) * 16));
        k_batch_radius<<<g2, 256, 0, s>>>(rowmax, row_cloud, total_pts, radius);
        TT_LAUNCH("k_batch_radius");
        const CloudTable T{pt_off, mat_off, sizes, bin_off, item_off};
        k_batch_hist<<<nchunks, kHistThreads, 0, s>>>(mats, T, chunks, radius, row_cnt, hist);
        TT_LAUNCH("k_batch_hist");
        scan_exclusive<u64>(&sctx, row_cnt, row_off, total_pts, reinterpret_cast<u64*>(count), 0);
        k_batch_bins<<<clouds, 1024, 0, s>>>(T, clouds, row_off, count, hist, bin_item, items, cursor, radix, edge_off);
        TT_LAUNCH("k_batch_bins");
        if (nparts)
            k_batch_part<<<nparts, kPartThreads, part_smem, s>>>(mats, T, parts, radius, radix, edge_off, bin_item,
                                                                 cursor, part_items, keys);
        TT_LAUNCH("k_batch_part");
        if (total_items)
            k_batch_items<<<total_items, kItemThreads, 0, s>>>(items, item_cloud, edge_off, keys, ed, ev);
        TT_LAUNCH("k_batch_items");
        // the marked clouds, each on its own (their keys are contiguous), by
        // the distance bits alone (stable: ties keep the index order): four
        // 8-bit passes
        const u32 g3 = u32(std::min<u64>((total_pts * 32 + 255) / 256, u64(owner->sms) * 32));
        k_batch_tiles<<<1, 1024, 0, s>>>(edge_off, radix, clouds, tile_place, seg_tiles, seg_ntiles);
        TT_LAUNCH("k_batch_tiles");
        k_batch_edges<<<g3, 256, 0, s>>>(mats, mat_off, sizes, pt_off, row_cloud, total_pts, radius, radix, ib, row_off,
                                         keys);
        TT_LAUNCH("k_batch_edges");
        const bool swapped =
            radix_sort_segments(&sctx, keys, kbuf, edge_off, seg_tiles, seg_ntiles, nseg_tiles, sure_tiles, seg_hist, 31,
                                ib);
        const u32 g4 = std::min<u32>(std::max<u32>(nseg_tiles, 1), u32(owner->sms) * 8);
        k_batch_emit<<<g4, 256, 0, s>>>(swapped ? kbuf : keys, edge_off, seg_tiles, seg_ntiles, ib, ed, ev);
        TT_LAUNCH("k_batch_emit");
        sctx.launches += 9;
    }

    static int bits_for(u64 v) {
        int b = 0;
        while ((1ull << b) < v) ++b;
        return b;
    }

    void release() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        for (void* q : owned) cudaFree(q);
        owned.clear();
        sctx.arena.release();
        if (sctx.stream) cudaStreamDestroy(sctx.stream);
        sctx.stream = nullptr;
    }
};

Batch* batch_create(tt_ctx* c, const u32* sizes_h, u32 clouds, u32 dim, int kind, f32 p, int use_graph) {
    if (clouds == 0) invalid("gb300: empty batch");
    if (dim == 0) invalid("gb300: dim must be >= 1");
    auto* b = new Batch;
    try {
        b->owner = c;
        b->clouds = clouds;
        b->dim = dim;
        b->kind = kind;
        b->p = p;
        b->use_graph = use_graph != 0;
        b->sctx.device = c->device;
        b->sctx.sms = c->sms;
        TT_CUDA(cudaStreamCreateWithFlags(&b->sctx.stream, cudaStreamNonBlocking));
        std::vector<u64> pt_off(clouds + 1, 0), mat_off(clouds + 1, 0);
        std::vector<Tile> tiles[kNumShapes];
        std::vector<u32> row_cloud;
        u64 pairs = 0;
        std::vector<Chunk> chunks;
        std::vector<Part> parts;
        u32 most_bins = 0;
        std::vector<u32> bin_off(clouds + 1, 0), item_off(clouds + 1, 0), item_cloud;
        for (u32 q = 0; q < clouds; ++q) {
            const u32 n = sizes_h[q];
            if (n < 1) invalid("gb300: every cloud needs at least one point");
            b->maxn = std::max(b->maxn, n);
            pt_off[q + 1] = pt_off[q] + n;
            mat_off[q + 1] = mat_off[q] + u64(n) * n;
            pairs += u64(n) * (n - 1) / 2;
            for (int si = 0; si < kNumShapes; ++si)   // the tiles on and above the diagonal
                for (u32 i0 = 0; i0 < n; i0 += u32(kShapes[si].r))
                    for (u32 j0 = i0; j0 < n; j0 += u32(kShapes[si].c)) tiles[si].push_back(Tile{q, i0, j0});
            for (u32 i = 0; i < n; ++i) row_cloud.push_back(q);
            // chunks of rows; bins of about 256 pairs (a power of two); items.
            // A cloud whose pairs, spread evenly, would overflow the most bins
            // there can be (5,018 points and more) goes to the radix sort at
            // once: one bin, no items.
            const u64 cp = u64(n) * (n - 1) / 2;
            u32 bins = cp <= u64(kMaxBins) * kBinMax ? 64 : 1;
            while (bins > 1 && bins < kMaxBins && u64(bins) * 256 < cp) bins *= 2;
            for (u32 i0 = 0; i0 < n;) {
                u32 i1 = i0;
                for (u64 held = 0; i1 < n && held < kChunkPairs; ++i1) held += i1;
                chunks.push_back(Chunk{q, i0, i1});
                i0 = i1;
            }
            if (bins > 1) {
                for (u64 i0 = 0; i0 < cp; i0 += kPartPairs) parts.push_back(Part{q, u32(i0)});
                most_bins = std::max(most_bins, bins);
            }
            bin_off[q + 1] = bin_off[q] + bins;
            const u32 cap = bins > 1 ? u32(cp / kItemStep) + 1 : 0;
            item_off[q + 1] = item_off[q] + cap;
            b->part_items = std::max(b->part_items, std::min(cap, bins));
            item_cloud.insert(item_cloud.end(), cap, q);
        }
        // the segmented sort's capacity: every cloud's largest key count
        // (every pair kept) in tiles of kSegTileKeys, 256 digit counts a tile
        u64 seg_cap = 0;
        u64 sure = 0;   // ... of the clouds without items
        for (u32 q = 0; q < clouds; ++q) {
            const u64 t = div_up(u64(sizes_h[q]) * (sizes_h[q] - 1) / 2, u64(kSegTileKeys));
            seg_cap += t;
            if (item_off[q + 1] == item_off[q]) sure += t;
        }
        if (256 * seg_cap >= (1ull << 32)) invalid("gb300: batch too large for the segmented sort's counts");
        b->ib = std::max(1, Batch::bits_for(u64(b->maxn) * (b->maxn - 1) / 2 + 1));
        if (b->ib + 31 + Batch::bits_for(clouds) > 64)
            invalid("gb300: batch too large for 64-bit edge keys (clouds x largest cloud)");
        b->total_pts = pt_off[clouds];
        b->total_mat = mat_off[clouds];
        b->total_pairs = std::max<u64>(pairs, 1);
        b->x = b->alloc<f32>(b->total_pts * dim);
        b->mats = b->alloc<f32>(b->total_mat);
        b->rowmax = b->alloc<u32>(b->total_pts);
        b->radius = b->alloc<u32>(clouds);
        b->pt_off = b->alloc<u64>(clouds + 1);
        b->mat_off = b->alloc<u64>(clouds + 1);
        b->sizes = b->alloc<u32>(clouds);
        for (int si = 0; si < kNumShapes; ++si) {
            b->ntiles[si] = u32(tiles[si].size());
            b->tiles[si] = b->alloc<Tile>(tiles[si].size());
        }
        b->row_cloud = b->alloc<u32>(row_cloud.size());
        b->next = b->alloc<u32>(1);
        b->keys = b->alloc<u64>(b->total_pairs);
        b->kbuf = b->alloc<u64>(b->total_pairs);
        b->row_cnt = b->alloc<u64>(b->total_pts);
        b->row_off = b->alloc<u64>(b->total_pts);
        b->count = b->alloc<unsigned long long>(1);
        b->nchunks = u32(chunks.size());
        b->chunks = b->alloc<Chunk>(chunks.size());
        b->total_bins = bin_off[clouds];
        b->bin_off = b->alloc<u32>(clouds + 1);
        b->hist = b->alloc<u32>(b->total_bins);
        b->bin_item = b->alloc<u16>(b->total_bins);
        b->nparts = u32(parts.size());
        b->parts = b->alloc<Part>(parts.size());
        b->part_smem = 8 * size_t(kPartPairs) + 8 * size_t(b->part_items) + 2 * size_t(most_bins);
        TT_CUDA(cudaFuncSetAttribute(k_batch_part, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPartSmemMax)));
        b->total_items = item_off[clouds];
        b->item_off = b->alloc<u32>(clouds + 1);
        b->items = b->alloc<Item>(b->total_items);
        b->cursor = b->alloc<u32>(b->total_items);
        b->item_cloud = b->alloc<u32>(b->total_items);
        b->radix = b->alloc<u32>(clouds);
        b->edge_off = b->alloc<u64>(clouds + 1);
        b->nseg_tiles = u32(seg_cap);
        b->sure_tiles = u32(sure);
        b->tile_place = b->alloc<uint2>(clouds);
        b->seg_hist = 256 * seg_cap;
        b->seg_tiles = b->alloc<SegTile>(seg_cap);
        b->seg_ntiles = b->alloc<u32>(1);
        b->ed = b->alloc<f32>(b->total_pairs);
        b->ev = b->alloc<int32_t>(2 * b->total_pairs);
        cudaStream_t s = b->sctx.stream;
        TT_CUDA(cudaMemcpyAsync(b->pt_off, pt_off.data(), 8 * (clouds + 1), cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->mat_off, mat_off.data(), 8 * (clouds + 1), cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->sizes, sizes_h, 4 * clouds, cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->chunks, chunks.data(), sizeof(Chunk) * chunks.size(), cudaMemcpyHostToDevice, s));
        if (!parts.empty())
            TT_CUDA(cudaMemcpyAsync(b->parts, parts.data(), sizeof(Part) * parts.size(), cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->bin_off, bin_off.data(), 4 * (clouds + 1), cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->item_off, item_off.data(), 4 * (clouds + 1), cudaMemcpyHostToDevice, s));
        if (!item_cloud.empty())
            TT_CUDA(cudaMemcpyAsync(b->item_cloud, item_cloud.data(), 4 * item_cloud.size(), cudaMemcpyHostToDevice, s));
        for (int si = 0; si < kNumShapes; ++si)
            TT_CUDA(cudaMemcpyAsync(b->tiles[si], tiles[si].data(), sizeof(Tile) * tiles[si].size(),
                                    cudaMemcpyHostToDevice, s));
        TT_CUDA(cudaMemcpyAsync(b->row_cloud, row_cloud.data(), 4 * row_cloud.size(), cudaMemcpyHostToDevice, s));
        // size the sort's and the row scan's scratch outside any capture
        radix_reserve_entries(&b->sctx, b->seg_hist);
        // the row scan's levels (64-bit entries: four times as many 32-bit
        // entries reserve at least their bytes at every level)
        radix_reserve_entries(&b->sctx, 4 * b->total_pts);
        TT_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        b->release();
        delete b;
        throw;
    }
    return b;
}

void batch_run(Batch* b) {
    if (!b->tuned) {   // the first run: pick the tile shape on this batch's points
        b->tune();
        b->tuned = true;
    }
    if (!b->use_graph) {
        const u64 before = b->sctx.launches;
        b->enqueue();
        b->graph_kernels = b->sctx.launches - before;
        return;
    }
    if (!b->exec) {
        TT_CUDA(cudaStreamBeginCapture(b->sctx.stream, cudaStreamCaptureModeThreadLocal));
        try {
            const u64 before = b->sctx.launches;
            b->enqueue();
            b->graph_kernels = b->sctx.launches - before;
        } catch (...) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(b->sctx.stream, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        TT_CUDA(cudaStreamEndCapture(b->sctx.stream, &b->graph));
        TT_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
    }
    TT_CUDA(cudaGraphLaunch(b->exec, b->sctx.stream));
}

}  // namespace tt

using namespace tt;

extern "C" {

int tt_batch_create(tt_ctx* c, const uint32_t* sizes, uint32_t count, uint32_t dim, int kind, float p,
                    int use_graph, tt_batch** out) {
    if (!c || !out) return TT_ERR_INVALID;
    try {
        TT_CUDA(cudaSetDevice(c->device));
        if (kind < TT_METRIC_L1 || kind > TT_METRIC_LP) invalid("metric: unknown kind");
        if (kind == TT_METRIC_LP && !(p >= 1.0f)) invalid("metric: p must be in [1, inf]");
        *out = reinterpret_cast<tt_batch*>(batch_create(c, sizes, count, dim, kind, p, use_graph));
        return TT_OK;
    } catch (const Error& e) {
        c->last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        c->last_error = e.what();
        return TT_ERR_INTERNAL;
    }
}

float* tt_batch_points(tt_batch* b) { return b ? reinterpret_cast<Batch*>(b)->x : nullptr; }

int tt_batch_tuning(tt_batch* bh, uint32_t* tile_rows, uint32_t* tile_cols, float* shape_ms, uint32_t* shapes,
                    int* from_cache) {
    Batch* b = reinterpret_cast<Batch*>(bh);
    if (!b) return TT_ERR_INVALID;
    if (tile_rows) *tile_rows = u32(kShapes[b->shape].r);
    if (tile_cols) *tile_cols = u32(kShapes[b->shape].c);
    if (shapes) *shapes = u32(kNumShapes);
    if (shape_ms)
        for (int si = 0; si < kNumShapes; ++si) shape_ms[si] = b->tune_ms[si];
    if (from_cache) *from_cache = b->tuned_from_cache ? 1 : 0;
    return TT_OK;
}

int tt_batch_run(tt_batch* bh, int wait) {
    Batch* b = reinterpret_cast<Batch*>(bh);
    if (!b) return TT_ERR_INVALID;
    try {
        TT_CUDA(cudaSetDevice(b->owner->device));
        batch_run(b);
        b->owner->launches += b->graph_kernels;   // the kernels one run launches
        if (wait) TT_CUDA(cudaStreamSynchronize(b->sctx.stream));
        return TT_OK;
    } catch (const Error& e) {
        b->owner->last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        b->owner->last_error = e.what();
        return TT_ERR_INTERNAL;
    }
}

int tt_batch_result(tt_batch* bh, tt_batch_out* out) {
    Batch* b = reinterpret_cast<Batch*>(bh);
    if (!b || !out) return TT_ERR_INVALID;
    out->clouds = b->clouds;
    out->total_points = b->total_pts;
    out->radius_dev = reinterpret_cast<const float*>(b->radius);
    out->edge_offset_dev = b->edge_off;
    out->diam_dev = b->ed;
    out->verts_dev = b->ev;
    out->mats_dev = b->mats;
    out->stream = b->sctx.stream;
    return TT_OK;
}

void tt_batch_destroy(tt_batch* bh) {
    Batch* b = reinterpret_cast<Batch*>(bh);
    if (!b) return;
    cudaSetDevice(b->owner->device);
    if (b->sctx.stream) cudaStreamSynchronize(b->sctx.stream);
    b->release();
    delete b;
}

}  // extern "C"
