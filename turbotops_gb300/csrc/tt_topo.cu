// tt_topo.cu — persistence pairs with their critical edges for a batch of
// clouds, and the adjoint that scatters dL/d(birth, death) onto coordinates.
//
// No counterpart in the reference (its Barcode keeps values only,
// rips.hpp:52-67). Forward: for every cloud the GPU runs the dense front end
// (distances, enclosing radius, dim0); host threads reduce dimension 1 of the
// clouds whose front end is done while the GPU works on the next ones (by
// columns, long ones by sweeps over the sorted edges: compute_pairs),
// recording each bar's critical simplices; each bar value is then the length
// of one edge:
//   H0 death   the spanning-tree edge that merged two components
//   H1 birth   the column's edge
//   H1 death   the longest edge of the pivot triangle (the edge whose length
//              equals the death value; unique on tie-free input)
// Adjoint: dL/dx_u += g * dd(u,v)/dx_u, dL/dx_v -= the same, for every
// critical edge (u, v) with upstream gradient g, where for
//   L2   dd/dx_u = (x_u - x_v) / d
//   L1   sign(x_u - x_v)
//   Linf e_k* sign(x_u,k* - x_v,k*), k* the first coordinate of largest |diff|
//   Lp   sign(diff_k) (|diff_k| / d)^(p - 1)
// one thread per edge, float atomics into the gradient.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstdlib>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "tt_internal.cuh"
#include "tt_metric.cuh"
#include "tt_reduce.h"

namespace tt {

namespace {

constexpr u32 NOV = 0xffffffffu;

__global__ void k_topo_adjoint(const f32* __restrict__ x, u32 dim, int kind, f32 p, const u32* __restrict__ edges,
                               const f32* __restrict__ g, u64 m, f32* __restrict__ grad) {
    for (u64 e = u64(blockIdx.x) * blockDim.x + threadIdx.x; e < m; e += u64(gridDim.x) * blockDim.x) {
        const u32 u = edges[2 * e], v = edges[2 * e + 1];
        const f32 ge = g[e];
        if (u == NOV || v == NOV || ge == 0.0f || u == v) continue;
        const f32* xu = x + u64(u) * dim;
        const f32* xv = x + u64(v) * dim;
        f32 s = 0.0f, mx = 0.0f;
        u32 kmax = 0;
        for (u32 k = 0; k < dim; ++k) {
            const f32 d = xu[k] - xv[k];
            const f32 a = fabsf(d);
            if (a > mx) {
                mx = a;
                kmax = k;
            }
            if (kind == M_L2) s = fmaf(d, d, s);
            else if (kind == M_LP) s += powf(a, p);
        }
        f32 dd = kind == M_L2 ? sqrtf(s) : kind == M_LP ? powf(s, 1.0f / p) : 0.0f;
        if ((kind == M_L2 || kind == M_LP) && !(dd > 0.0f)) continue;
        for (u32 k = 0; k < dim; ++k) {
            const f32 d = xu[k] - xv[k];
            f32 w;
            if (kind == M_L2) w = d / dd;
            else if (kind == M_L1) w = d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f);
            else if (kind == M_LINF) w = k == kmax ? (d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f)) : 0.0f;
            else w = (d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f)) * powf(fabsf(d) / dd, p - 1.0f);
            if (w != 0.0f) {
                atomicAdd(&grad[u64(u) * dim + k], ge * w);
                atomicAdd(&grad[u64(v) * dim + k], -ge * w);
            }
        }
    }
}

void decode2(u64 idx, u32& a, u32& b) {   // a > b
    u64 v = u64((1.0 + std::sqrt(1.0 + 8.0 * double(idx))) * 0.5);
    while (v * (v - 1) / 2 > idx) --v;
    while ((v + 1) * v / 2 <= idx) ++v;
    a = u32(v);
    b = u32(idx - v * (v - 1) / 2);
}

void decode3(u64 idx, u32 n, u32& c0, u32& c1, u32& c2) {   // c0 > c1 > c2
    u32 lo = 2, hi = n;
    while (hi - lo > 1) {   // largest v with C(v, 3) <= idx
        const u32 mid = lo + (hi - lo) / 2;
        if (u64(mid) * (mid - 1) * (mid - 2) / 6 <= idx) lo = mid;
        else hi = mid;
    }
    c0 = lo;
    decode2(idx - u64(lo) * (lo - 1) * (lo - 2) / 6, c1, c2);
}

// A cloud's outputs on the host: in the context's page-locked staging (the
// copies are then asynchronous and touch no fresh pages), or, past its limit,
// in memory of their own.
template <typename T>
struct Out {
    T* p = nullptr;
    u64 count = 0;
    std::vector<T> own;
    T* data() { return p; }
    const T* data() const { return p; }
    u64 size() const { return count; }
    const T& operator[](u64 i) const { return p[i]; }
};

struct Cloud {
    u32 n = 0;
    u64 off = 0;
    f32 thr = 0;
    Out<f32> mat, h0d, cd;
    Out<u64> h0e, ci, emi, keys;
    Out<u8> emf;
    host::Bars bars;
};

constexpr u64 kStagingMax = u64(256) << 20;

// The bytes of staging a cloud's outputs may take: matrix and keys, H0, a few
// columns a point.
u64 staging_bytes(u64 n) { return 8 * n * n + 256 * n + 1024; }

// Takes a cloud's outputs off the device, into its part of the staging.
struct Staging {
    cudaStream_t stream;
    unsigned char* base;
    u64 left;
    template <typename T>
    void take(Out<T>& o, const T* dev, u64 count) {
        o.count = count;
        const u64 bytes = (count * sizeof(T) + 15) & ~u64(15);
        if (bytes <= left) {
            o.p = reinterpret_cast<T*>(base);
            base += bytes;
            left -= bytes;
        } else {
            o.own.resize(count);
            o.p = o.own.data();
        }
        if (count) TT_CUDA(cudaMemcpyAsync(o.p, dev, count * sizeof(T), cudaMemcpyDeviceToHost, stream));
    }
};

// The front end of a cloud of a few hundred points is a chain of some 25 small
// kernels and two waits, so the clouds' chains run on kLanes streams, each with
// a context (workspaces) of its own and driven by its own thread. A gradient
// step over 64 clouds of 100 points 13.4 ms with one lane, 6.9 with four, 5.3
// with six, 4.6 with eight; of 512 points 21.6, 17.5, 17.5 and 17.5 (the
// reductions then take the time, and need the threads); 12 of 2,048 points 86, 79,
// 79 and 79 ms. Larger clouds fill the chip by themselves (6 of 3,000 points 218
// ms either way), and their workspaces are not held several times. Two clouds gain
// nothing (2 x 300 points 2.46 ms, two lanes 2.56; 3 x 256 points 2.37 and 2.29).
// The lanes' contexts (up to 130 MB each at 2,048 points) and the staging stay
// with the caller's context and are given back with it.
constexpr u32 kLanes = 6;
constexpr u32 kLaneMaxN = 2048;

tt_ctx* lane_context(tt_ctx* c, u32 lane) {   // lane >= 1; kept by c
    while (c->lanes.size() < lane) {
        auto* l = new tt_ctx;
        c->lanes.push_back(l);
        l->device = c->device;
        l->sms = c->sms;
        l->own_stream = true;
        TT_CUDA(cudaStreamCreateWithFlags(&l->stream, cudaStreamNonBlocking));
    }
    if (!c->lanes[lane - 1]->stream) TT_CUDA(cudaStreamCreateWithFlags(&c->lanes[lane - 1]->stream, cudaStreamNonBlocking));
    return c->lanes[lane - 1];
}

// Hands clouds from the threads that run their device front ends to the
// threads that reduce them: a cloud is published once its outputs are on the
// host, and reducers take clouds in the order they were published, so the
// reductions of the first clouds overlap the front end of the later ones and a
// thread that finishes early takes the next cloud. Each cloud's reduction is
// independent of the others, so the bars do not depend on the schedule.
struct CloudQueue {
    std::mutex m;
    std::condition_variable cv;
    std::vector<u32> ready;
    size_t next = 0, expected;
    bool stop = false;
    explicit CloudQueue(size_t e) : expected(e) {}
    // the next cloud to reduce; NOV when none is left (or after stop)
    u32 take() {
        std::unique_lock<std::mutex> lk(m);
        cv.wait(lk, [&] { return stop || next < ready.size() || next >= expected; });
        if (stop || next >= expected) return NOV;
        const u32 q = ready[next++];
        if (next >= expected) cv.notify_all();   // none is left for those that wait
        return q;
    }
    void publish(u32 q) {
        {
            std::lock_guard<std::mutex> lk(m);
            ready.push_back(q);
        }
        cv.notify_all();
    }
    void halt() {
        {
            std::lock_guard<std::mutex> lk(m);
            stop = true;
        }
        cv.notify_all();
    }
    bool halted() {
        std::lock_guard<std::mutex> lk(m);
        return stop;
    }
};

}  // namespace

struct TopoResult {
    tt_topo_out pub{};
    std::vector<u64> h0_off, h1_off;
    std::vector<f32> h0_death, h1_birth, h1_death;
    std::vector<u32> h0_edge, h1_bedge, h1_dedge;
};

}  // namespace tt

using namespace tt;

extern "C" int tt_topo_forward(tt_ctx* c, const float* x, const uint32_t* sizes, uint32_t count, uint32_t dim,
                               int kind, float p, int threads, tt_topo_out** out) {
    if (!c || !out) return TT_ERR_INVALID;
    *out = nullptr;
    try {
        TT_CUDA(cudaSetDevice(c->device));
        if (kind < TT_METRIC_L1 || kind > TT_METRIC_LP) invalid("metric: unknown kind");
        if (kind == TT_METRIC_LP && !(p >= 1.0f)) invalid("metric: p must be in [1, inf]");
        std::vector<Cloud> cl(count);
        u64 points = 0;
        u32 maxn = 0, clouds = 0;
        for (u32 q = 0; q < count; ++q) {
            cl[q].n = sizes[q];
            cl[q].off = points;
            points += sizes[q];
            maxn = std::max(maxn, sizes[q]);
            clouds += sizes[q] > 0;
        }
        // host reducers (the calling thread and the other front-end threads
        // join them after the front end)
        u32 nt = threads > 0 ? u32(threads) : std::max(1u, std::thread::hardware_concurrency());
        // threads beyond one per cloud go into each cloud's own reduction
        const unsigned per_cloud = count ? std::max<u32>(1, nt / std::max<u32>(count, 1)) : 1;
        nt = std::min<u32>(nt, std::max<u32>(count, 1));
        const u32 lanes = maxn <= kLaneMaxN && clouds > 2 ? std::min(nt, kLanes) : 1;
        std::vector<tt_ctx*> lane(lanes, c);
        for (u32 l = 1; l < lanes; ++l) lane[l] = lane_context(c, l);
        // every cloud's part of the staging
        u64 want = 0;
        for (u32 q = 0; q < count; ++q) want += staging_bytes(cl[q].n);
        u64 staged = std::min(want, kStagingMax);
        unsigned char* staging = nullptr;
        if (staged) try {
                staging = static_cast<unsigned char*>(c->staging.get(staged));
            } catch (const Error&) {   // (no page-locked memory left: the clouds' own)
                cudaGetLastError();
                staged = 0;
            }
        std::vector<Staging> out_of(count);
        u64 at = 0;
        for (u32 q = 0; q < count; ++q) {
            const u64 bytes = staging_bytes(cl[q].n) & ~u64(15);
            const bool fits = at + bytes <= staged;
            out_of[q] = Staging{nullptr, fits ? staging + at : nullptr, fits ? bytes : 0};
            if (fits) at += bytes;
        }
        CloudQueue queue(clouds);
        std::vector<std::exception_ptr> errs(nt);
        auto reduce = [&](Cloud& C) {
            std::vector<host::Entry> cols(C.ci.size());
            for (u64 i = 0; i < cols.size(); ++i) cols[i] = host::Entry{C.ci[i], C.cd[i]};
            host::HostComplex hc{C.mat.data(), nullptr, nullptr, nullptr, C.n, C.thr};
            std::vector<u64> piv;
            host::ReduceStats st;
            try {
                const host::SortedEdges edges{[&] { return C.keys.data(); }, C.keys.size()};
                C.bars = host::compute_pairs(hc, 1, 1, cols, C.emi.data(), C.emf.data(), piv, st, per_cloud, &edges);
            } catch (const std::exception& e) {
                throw Error(TT_ERR_INTERNAL, e.what());
            }
        };
        // device front end of a lane's clouds; each cloud goes to the reducers
        // once its outputs are on the host
        std::atomic<u32> next{0};
        auto front_end = [&](tt_ctx* lc) {
            u32 before = NOV;
            for (u32 q; (q = next.fetch_add(1)) < count && !queue.halted();) {
                Cloud& C = cl[q];
                if (C.n == 0) continue;
                const u32 n = C.n;
                f32* mat = lc->arena.get<f32>(S_MAT, u64(n) * n + 1);
                C.thr = dense_radius(lc, x + C.off * dim, n, dim, kind, p, mat);
                Complex cx{mat, nullptr, nullptr, nullptr, n, C.thr};
                // (the radius has just been waited for, and with it the copies of the lane's cloud before)
                if (before != NOV) queue.publish(before);
                Dim0Out r;
                dim0(lc, cx, 1, r);
                Staging st = out_of[q];
                st.stream = lc->stream;
                st.take(C.mat, mat, u64(n) * n);
                st.take(C.keys, r.keys, n <= host::kSweepMaxN ? r.m : 0);
                st.take(C.h0d, r.h0, r.nh0);
                st.take(C.h0e, r.h0_edge, r.nh0);
                st.take(C.ci, r.cidx, r.ncols);
                st.take(C.cd, r.cd, r.ncols);
                st.take(C.emi, r.emi, r.ncols);
                st.take(C.emf, r.emf, r.ncols);
                before = q;
            }
            TT_CUDA(cudaStreamSynchronize(lc->stream));
            if (before != NOV) queue.publish(before);
        };
        auto work = [&](u32 t) {   // of thread t: its lane, then the reductions
            try {
                if (t < lanes) {
                    TT_CUDA(cudaSetDevice(c->device));
                    front_end(lane[t]);
                }
                for (u32 q; (q = queue.take()) != NOV;) reduce(cl[q]);
            } catch (...) {
                errs[t] = std::current_exception();
                queue.halt();
                if (t < lanes) cudaStreamSynchronize(lane[t]->stream);   // no copy outlives its target
            }
        };
        // the other lanes' streams follow the caller's
        if (lanes > 1) {
            cudaEvent_t ev;
            TT_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            cudaError_t e = cudaEventRecord(ev, c->stream);
            for (u32 l = 1; l < lanes && e == cudaSuccess; ++l) e = cudaStreamWaitEvent(lane[l]->stream, ev, 0);
            cudaEventDestroy(ev);
            TT_CUDA(e);
        }
        std::vector<u64> launched(lanes);
        for (u32 l = 0; l < lanes; ++l) launched[l] = lane[l]->launches;
        std::vector<std::thread> pool;
        try {
            for (u32 t = 1; t < nt; ++t) pool.emplace_back(work, t);
        } catch (...) {
            queue.halt();
            for (auto& th : pool) th.join();
            throw;
        }
        work(0);
        for (auto& th : pool) th.join();
        for (u32 l = 1; l < lanes; ++l) c->launches += lane[l]->launches - launched[l];
        for (auto& e : errs)
            if (e) std::rethrow_exception(e);
        // pack, with global point ids
        auto* R = new TopoResult;
        R->h0_off.assign(count + 1, 0);
        R->h1_off.assign(count + 1, 0);
        for (u32 q = 0; q < count; ++q) {
            const Cloud& C = cl[q];
            for (u64 i = 0; i < C.h0d.size(); ++i) {
                u32 a, b;
                decode2(C.h0e[i], a, b);
                R->h0_death.push_back(C.h0d[i]);
                R->h0_edge.push_back(u32(C.off + a));
                R->h0_edge.push_back(u32(C.off + b));
            }
            R->h0_off[q + 1] = R->h0_death.size();
            for (u64 i = 0; i < C.bars.birth.size(); ++i) {
                u32 a, b;
                decode2(C.bars.birth_idx[i], a, b);
                R->h1_birth.push_back(C.bars.birth[i]);
                R->h1_death.push_back(C.bars.death[i]);
                R->h1_bedge.push_back(u32(C.off + a));
                R->h1_bedge.push_back(u32(C.off + b));
                u32 du = NOV, dv = NOV;
                if (C.bars.death_idx[i] != kNone) {
                    u32 c0, c1, c2;
                    decode3(C.bars.death_idx[i], C.n, c0, c1, c2);
                    const f32 dd = C.bars.death[i];
                    const f32* M = C.mat.data();
                    if (M[u64(c1) * C.n + c2] == dd) { du = c1; dv = c2; }
                    else if (M[u64(c0) * C.n + c2] == dd) { du = c0; dv = c2; }
                    else { du = c0; dv = c1; }
                    du = u32(C.off + du);
                    dv = u32(C.off + dv);
                }
                R->h1_dedge.push_back(du);
                R->h1_dedge.push_back(dv);
            }
            R->h1_off[q + 1] = R->h1_birth.size();
        }
        tt_topo_out& P = R->pub;
        P.clouds = count;
        P.h0_offset = R->h0_off.data();
        P.h0_death = R->h0_death.data();
        P.h0_edge = R->h0_edge.data();
        P.h1_offset = R->h1_off.data();
        P.h1_birth = R->h1_birth.data();
        P.h1_death = R->h1_death.data();
        P.h1_birth_edge = R->h1_bedge.data();
        P.h1_death_edge = R->h1_dedge.data();
        P.opaque = R;
        *out = &R->pub;
        return TT_OK;
    } catch (const Error& e) {
        c->last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        c->last_error = e.what();
        return TT_ERR_INTERNAL;
    }
}

extern "C" void tt_topo_free(tt_topo_out* out) {
    if (!out) return;
    delete static_cast<TopoResult*>(out->opaque);
}

extern "C" int tt_topo_adjoint(tt_ctx* c, const float* x, uint32_t dim, int kind, float p, const uint32_t* edges,
                               const float* grad_d, uint64_t m, float* grad_x) {
    if (!c) return TT_ERR_INVALID;
    try {
        TT_CUDA(cudaSetDevice(c->device));
        if (kind < TT_METRIC_L1 || kind > TT_METRIC_LP) invalid("metric: unknown kind");
        if (m) {
            const u32 grid = u32(std::min<u64>((m + 255) / 256, u64(c->sms) * 16));
            k_topo_adjoint<<<grid, 256, 0, c->stream>>>(x, dim, kind, p, edges, grad_d, m, grad_x);
            TT_LAUNCH("k_topo_adjoint");
            ++c->launches;
        }
        return TT_OK;
    } catch (const Error& e) {
        c->last_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        c->last_error = e.what();
        return TT_ERR_INTERNAL;
    }
}
