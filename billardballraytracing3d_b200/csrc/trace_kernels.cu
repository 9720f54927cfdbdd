// Trace-path kernels for sm_100a: BVH query, SurfacePatch stage 1 + Newton,
// and the bounce loop with reflection and nudge, all in exact FP64.
//
// Compiled with -fmad=false: every FP64 decision equals the reference's
// (see exact.cuh).  The wavefront's Newton kernels, its round control, the
// per-thread tail, single queries by brute force or on one object, and the
// drivers' ray generation and reductions; rounds are in advance.cu, warp-per-ray
// traces and queries in ray_warp.cu.
//
// Reference (manuelarturosantana/BillardBallRayTracing3D):
//   RayTracingDriver::trace_ray   include/RayTracingDriver.hpp:172-242
//   BVH::intersect                include/BVH.hpp:75-128
//   SurfacePatch::intersect       include/ScatObjects/SurfacePatch.hpp:253-303
//   Triangle::intersect           include/ScatObjects/Triangle.hpp:26-28
//   brute_force_intersect         include/BruteForce.hpp:7-16
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <mutex>

#include "trace_common.cuh"
#include "newton_group.cuh"

namespace bbrt {

cudaError_t launch_rays(const DScene& S, const TraceArgs& A, const WaveArgs& W, const NewtonRequest* reqs, const int* rays,
                        long long n, int sm_count, cudaStream_t stream);
cudaError_t rays_prepare();

// Newton on patch pidx in the scene's precision mode.
__device__ __forceinline__ int newton_mode(const DScene& S, int pidx, const V3& o, const V3& d, double u, double v,
                                           double t, QHit& h, long long& iters, long long& iters32) {
    if (S.precision == BBRT_PREC_SPLIT) return newton_split(S, pidx, o, d, u, v, t, h, iters, iters32);
    return newton_exact(S, pidx, o, d, u, v, t, h, iters);
}

// Newton solves of one round, one request per thread.  With a learned guess,
// a confident guess is tried first; its root is kept only when it converges
// inside the patch within guess_t_window patch sizes of the stage-1 t, and
// otherwise the solve restarts from the stage-1 triangle (the reference's start).
__device__ __forceinline__ void newton_thread_body(const DScene& S, const TraceArgs& A, const WaveArgs& W,
                                                   long long n_req) {
    if (blockIdx.x * static_cast<long long>(blockDim.x) >= n_req) return;   // graph launch: spare blocks
    const long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    long long iters = 0, iters32 = 0, used = 0, fallback = 0, off = 0;
    if (j < n_req) {
        const NewtonRequest q = W.req[j];
        if (W.next_req) W.next_req[j] = q;
        const V3 o = load3(W.o + 3LL * q.ray);
        const V3 d = load3(W.d + 3LL * q.ray);
        const int pidx = S.obj_sub[q.obj];
        QHit h;
        h.err = 0;
        h.ev0 = h.ev1 = 0.0;
        h.t = 0.0;
        h.p = h.n = v3(0.0, 0.0, 0.0);
        h.u = h.v = 0.0;
        // One solve for every request, from the guess where it is confident
        // (one call site, so requests of both kinds in a warp run together);
        // a second solve from the triangle only for abandoned guesses.
        double su, sv, st;
        key_to_uv(S, q.key, su, sv);
        st = q.t0;
        double win = 0.0;
        if (W.guess) {
            const double* g = W.guess + 4 * j;
            win = W.guess_t_window * W.frame[16LL * pidx + 12];
            if (g[3] > W.guess_min_logit && isfinite(g[0]) && isfinite(g[1]) && fabs(g[2] - q.t0) <= win) {
                used = 1;
                su = g[0];
                sv = g[1];
                st = g[2];
            }
        }
        const QHit h0 = h;
        CountersT<false> dummy;
        const int ok = S.obj_kind[q.obj] == BBRT_OBJ_PATCH ? newton_mode(S, pidx, o, d, su, sv, st, h, iters, iters32)
                                                           : triangle_intersect(S, pidx, o, d, h, dummy);
        if (used && !(ok && fabs(h.t - q.t0) <= win)) {
            fallback = 1;
            h = h0;
            double u0, v0;
            key_to_uv(S, q.key, u0, v0);
            newton_mode(S, pidx, o, d, u0, v0, q.t0, h, iters, iters32);
        }
        if (A.off_patch_miss && h.err == BBRT_RAY_NEWTON_DOMAIN &&
            !guess_inside(W.guess ? W.guess + 4 * j : nullptr, W.guess_min_logit)) {
            off = 1;   // not hit: resolved with t = +inf
            h.err = 0;
            h.t = CUDART_INF;
        }
        if (A.samples && h.err == 0) record_sample(A, 1, o, d, pidx, h.u, h.v, h.t);
        // a root outside the patch teaches the network a miss near the edge
        if (A.samples && h.err == BBRT_RAY_NEWTON_DOMAIN) record_sample(A, 0, o, d, pidx, 0.0, 0.0, 0.0);
        const long long e = static_cast<long long>(q.ray) * W.results + (q.entry & (W.results - 1));
        double* rd = W.res_data + e * kResData;
        rd[0] = h.t; rd[1] = h.p.x; rd[2] = h.p.y; rd[3] = h.p.z;
        rd[4] = h.n.x; rd[5] = h.n.y; rd[6] = h.n.z; rd[7] = h.u; rd[8] = h.v; rd[9] = h.ev0; rd[10] = h.ev1;
        W.res_err[e] = h.err;
        if (A.ray_work) A.ray_work[4LL * q.ray + 3] += iters + iters32;
    }
    if (A.stats) {
        warp_add(A.stats + ST_NEWTON_ITERS, iters);
        warp_add(A.stats + ST_NEWTON_ITERS_FP32, iters32);
        warp_add(A.stats + ST_GUESS_USED, used);
        warp_add(A.stats + ST_GUESS_FALLBACK, fallback);
        warp_add(A.stats + ST_OFF_PATCH, off);
    }
}

// k_newton with 8 lanes per request (patches of at most 8 nodes per axis):
// the same starts, fallbacks and results, bit for bit.
__device__ __forceinline__ void newton_grp_body(const DScene& S, const TraceArgs& A, const WaveArgs& W,
                                                long long n_req) {
    if (blockIdx.x * static_cast<long long>(blockDim.x) / kGroup >= n_req) return;   // graph launch: spare blocks
    const Grp G = make_grp();
    const long long j = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) / kGroup;
    long long iters = 0, iters32 = 0, used = 0, fallback = 0, off = 0;
    if (j < n_req) {   // uniform over the group
        const NewtonRequest q = W.req[j];
        if (W.next_req && G.g == 0) W.next_req[j] = q;
        const V3 o = load3(W.o + 3LL * q.ray);
        const V3 d = load3(W.d + 3LL * q.ray);
        const int pidx = S.obj_sub[q.obj];
        QHit h;
        h.err = 0;
        h.ev0 = h.ev1 = 0.0;
        h.t = 0.0;
        h.p = h.n = v3(0.0, 0.0, 0.0);
        h.u = h.v = 0.0;
        bool done = false;
        if (W.guess) {
            const double* g = W.guess + 4 * j;
            const double win = W.guess_t_window * W.frame[16LL * pidx + 12];
            if (g[3] > W.guess_min_logit && isfinite(g[0]) && isfinite(g[1]) && fabs(g[2] - q.t0) <= win) {
                used = 1;
                QHit hg = h;
                if (grp_newton_mode(S, pidx, o, d, g[0], g[1], g[2], hg, iters, iters32, G) &&
                    fabs(hg.t - q.t0) <= win) {
                    h = hg;
                    done = true;
                } else {
                    fallback = 1;
                }
            }
        }
        if (S.obj_kind[q.obj] != BBRT_OBJ_PATCH) {
            CountersT<false> dummy;
            triangle_intersect(S, pidx, o, d, h, dummy);
        } else if (!done) {
            double u0, v0;
            key_to_uv(S, q.key, u0, v0);
            grp_newton_mode(S, pidx, o, d, u0, v0, q.t0, h, iters, iters32, G);
        }
        if (A.off_patch_miss && h.err == BBRT_RAY_NEWTON_DOMAIN &&
            !guess_inside(W.guess ? W.guess + 4 * j : nullptr, W.guess_min_logit)) {
            off = 1;
            h.err = 0;
            h.t = CUDART_INF;
        }
        if (G.g == 0) {
            if (A.samples && h.err == 0) record_sample(A, 1, o, d, pidx, h.u, h.v, h.t);
            if (A.samples && h.err == BBRT_RAY_NEWTON_DOMAIN) record_sample(A, 0, o, d, pidx, 0.0, 0.0, 0.0);
            const long long e = static_cast<long long>(q.ray) * W.results + (q.entry & (W.results - 1));
            double* rd = W.res_data + e * kResData;
            rd[0] = h.t; rd[1] = h.p.x; rd[2] = h.p.y; rd[3] = h.p.z;
            rd[4] = h.n.x; rd[5] = h.n.y; rd[6] = h.n.z; rd[7] = h.u; rd[8] = h.v; rd[9] = h.ev0; rd[10] = h.ev1;
            W.res_err[e] = h.err;
            if (A.ray_work) A.ray_work[4LL * q.ray + 3] += iters + iters32;
        }
    }
    if (G.g != 0) iters = iters32 = used = fallback = off = 0;
    if (A.stats) {
        warp_add(A.stats + ST_NEWTON_ITERS, iters);
        warp_add(A.stats + ST_NEWTON_ITERS_FP32, iters32);
        warp_add(A.stats + ST_GUESS_USED, used);
        warp_add(A.stats + ST_GUESS_FALLBACK, fallback);
        warp_add(A.stats + ST_OFF_PATCH, off);
    }
}

__global__ void __launch_bounds__(128) k_newton(DScene S, TraceArgs A, WaveArgs W, long long n_req) {
    if (W.count_dev) n_req = *W.count_dev;
    newton_thread_body(S, A, W, n_req);
}

__global__ void __launch_bounds__(128) k_newton_grp(DScene S, TraceArgs A, WaveArgs W, long long n_req) {
    if (W.count_dev) n_req = *W.count_dev;
    newton_grp_body(S, A, W, n_req);
}

// A round's Newton solves with the solver picked by the round's size: one
// request per thread for a big round (throughput), 8 lanes per request for a
// small one (at most W.newton_group_max requests, and the grid has their
// lanes), whose time is its slowest solve's latency.  Same results bit for
// bit either way.
__global__ void __launch_bounds__(128, 4) k_newton_auto(DScene S, TraceArgs A, WaveArgs W, long long n_req) {
    if (W.count_dev) n_req = *W.count_dev;
    if (n_req <= W.newton_group_max && n_req * kGroup <= static_cast<long long>(gridDim.x) * blockDim.x)
        newton_grp_body(S, A, W, n_req);
    else
        newton_thread_body(S, A, W, n_req);
}

// Finishes rays from their saved state with inline queries (the tail of a
// wavefront trace, and rays whose query overflowed the resolved list), or the
// single queries of such a round.  The current query restarts from the root, so
// the result is the same.
__global__ void __launch_bounds__(128) k_resume(DScene S, TraceArgs A, WaveArgs W, const NewtonRequest* reqs,
                                                const int* rays, long long n) {
    if (W.count_dev) {
        n = *W.count_dev;
        if (blockIdx.x * static_cast<long long>(blockDim.x) >= n) return;   // graph launch: spare blocks
    }
    const long long slot = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    Counters ctr;
    RayTally tally;
    if (slot < n) {
        const long long i = reqs ? reqs[slot].ray : rays[slot];
        int nres;
        RayCtx r = load_ray(A, W, i, nres);
        if (A.query_out) {
            write_hit(static_cast<bbrt_hit*>(A.query_out) + i, bvh_query(S, r.o, r.d, A.cull, ctr, false, r.member));
        } else {
            run_ray(S, A, i, r, ctr, tally.queries);
            add_ray_work(A, i, ctr);
            finish_ray(A, i, r);
            tally.bounces += r.bounces;
            tally.hist[r.status]++;
        }
    }
    flush_stats(A, ctr, tally, true);
}

// One BVH query per thread.
template <bool PATCHES>
__global__ void __launch_bounds__(128) k_query_bvh(DScene S, QueryArgs Q) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= Q.n) return;
    CountersT<false> ctr;
    write_hit(static_cast<bbrt_hit*>(Q.out) + i,
              bvh_query<PATCHES>(S, load3(Q.origins + 3 * i), load3(Q.dirs + 3 * i), Q.cull, ctr));
}

// One query per thread: brute force over all objects, or one object.
__global__ void __launch_bounds__(128) k_query(DScene S, QueryArgs Q) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= Q.n) return;
    const V3 o = load3(Q.origins + 3 * i);
    const V3 d = load3(Q.dirs + 3 * i);
    Counters ctr;
    QHit r;
    r.obj = -1;
    r.err = 0;
    r.t = 0.0;
    r.p = r.n = v3(0.0, 0.0, 0.0);
    r.u = r.v = r.ev0 = r.ev1 = 0.0;
    const bool use_cull = cull_ok(S, -1, Q.cull, o, d);
    CullRay cr;
    if (use_cull) cr = make_cull_ray(S, -1, o, d);
    if (Q.mode == BBRT_QUERY_BRUTE) {
        bool have = false;
        for (int k = 0; k < S.n_objects; ++k) {
            QHit h;
            const int hit = object_intersect(S, k, o, d, use_cull, cr, h, ctr);
            if (h.err) { r = h; r.obj = k; have = false; break; }
            if (hit && (!have || h.t < r.t)) { r = h; r.obj = k; have = true; }
        }
        if (!have && !r.err) r.obj = -1;
    } else {
        QHit h;
        const int hit = object_intersect(S, Q.object, o, d, use_cull, cr, h, ctr);
        if (h.err) { r = h; r.obj = Q.object; }
        else if (hit) { r = h; r.obj = Q.object; }
    }
    write_hit(static_cast<bbrt_hit*>(Q.out) + i, r);
}

// ---- host launchers -------------------------------------------------------
// ---- allocation-free trace (bbrt_trace_noalloc) ----------------------------
//
// The trace kernel's scratch — its ray counter, its statistics block
// and per-object hit counters — lives in this file-scope device array
// instead of memory allocated per scene or per call: word 0 is the counter,
// words [1, 1 + ST_COUNT) the statistics, words [kNoAllocHeader,
// kNoAllocHeader + n_objects) the hit counters.  One copy exists per device
// that loads the library, for the life of the process.  Host code must not
// use the array's name as a device address; noalloc_scratch() returns the
// address the device sees.
constexpr int kNoAllocHeader = 32;
static_assert(1 + ST_COUNT <= kNoAllocHeader, "the statistics block would overlap the per-object hit counters");
static __device__ __align__(256) unsigned long long g_noalloc_scratch[kNoAllocHeader + BBRT_NOALLOC_MAX_OBJECTS];

// Device address of g_noalloc_scratch on the current device, looked up with
// cudaGetSymbolAddress the first time each device asks.
cudaError_t noalloc_scratch(unsigned long long** out) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static void* addr[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(mu);
    if (addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        addr[dev] = p;
    }
    *out = static_cast<unsigned long long*>(addr[dev]);
    return cudaSuccess;
}

// Loads, on the current device, everything bbrt_trace_noalloc needs from this
// module: the scratch array's address and the warp-per-ray kernels.  Under lazy
// module loading the first use of either would otherwise load the module
// (which allocates device memory, the array included) inside the first
// allocation-free call; bbrt_scene_upload calls this instead.
cudaError_t noalloc_prepare() {
    unsigned long long* p = nullptr;
    cudaError_t e = noalloc_scratch(&p);
    if (e != cudaSuccess) return e;
    return rays_prepare();
}

// The warp-per-ray trace with its scratch in g_noalloc_scratch.  Clears the
// words this call uses first, then traces; hit counters (when asked for) are
// copied to the caller's device array and the statistics to `host_stats`.
cudaError_t launch_trace_noalloc(const DScene& S, TraceArgs A, bool count_hits, long long* hit_counts_out,
                                 long long* host_stats, cudaStream_t stream, int sm_count) {
    unsigned long long* scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) return e;
    const size_t words = kNoAllocHeader + (count_hits ? static_cast<size_t>(S.n_objects) : 0);
    e = cudaMemsetAsync(scratch, 0, words * sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
    A.work_counter = scratch;
    A.stats = reinterpret_cast<long long*>(scratch + 1);
    A.hit_counts = count_hits ? scratch + kNoAllocHeader : nullptr;
    e = launch_rays(S, A, WaveArgs(), nullptr, nullptr, A.n, sm_count, stream);
    if (e != cudaSuccess) return e;
    if (count_hits) {
        e = cudaMemcpyAsync(hit_counts_out, scratch + kNoAllocHeader, sizeof(long long) * S.n_objects,
                            cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return e;
    }
    if (host_stats) {
        e = cudaMemcpyAsync(host_stats, scratch + 1, sizeof(long long) * ST_COUNT, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
        e = cudaStreamSynchronize(stream);
    }
    return e;
}

size_t wave_bytes_per_ray() {
    return sizeof(double) * 6 + sizeof(int) * 2 + sizeof(int) * 2 * kResolved + sizeof(double) * kResolved * kResData +
           2 * sizeof(NewtonRequest) + sizeof(int) + sizeof(int) * (kQsInt + kSaveStack) + sizeof(double);
}

// Carves the wavefront workspace for n rays out of `ws` (wave_bytes_per_ray() * n bytes).
void wave_layout(void* ws, long long n, WaveArgs& W, NewtonRequest*& req_a, NewtonRequest*& req_b) {
    char* p = static_cast<char*>(ws);
    auto take = [&](size_t bytes) { char* q = p; p += (bytes + 255) & ~static_cast<size_t>(255); return q; };
    W.o = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    W.d = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    W.bounces = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.nres = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.res_obj = reinterpret_cast<int*>(take(sizeof(int) * kResolved * n));
    W.res_err = reinterpret_cast<int*>(take(sizeof(int) * kResolved * n));
    W.res_data = reinterpret_cast<double*>(take(sizeof(double) * kResolved * kResData * n));
    req_a = reinterpret_cast<NewtonRequest*>(take(sizeof(NewtonRequest) * n));
    req_b = reinterpret_cast<NewtonRequest*>(take(sizeof(NewtonRequest) * n));
    W.overflow = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.qs_int = reinterpret_cast<int*>(take(sizeof(int) * kQsInt * n));
    W.qs_t = reinterpret_cast<double*>(take(sizeof(double) * n));
    W.qs_stack = reinterpret_cast<int*>(take(sizeof(int) * kSaveStack * n));
}

size_t wave_workspace_bytes(long long n) { return wave_bytes_per_ray() * n + 20 * 256; }


// Round control of the graph-launched trace, after each k_advance: the same
// decision the host-driven loop takes from the round's counters.  No requests,
// or a watchdog stop: the rounds end.  At most wave_tail requests: the rounds
// end and the tail kernel finishes those rays.  Otherwise the requests go to
// Newton and become the next round's runnable set; the loop repeats unless
// this was round max_rounds (flagged for the host as an error).  Every
// repetition raises counters[kWcRounds], so the loop ends after at most
// max_rounds rounds whatever the counts.
__global__ void k_wave_decide(unsigned int* c, long long wave_tail, long long max_rounds,
                              cudaGraphConditionalHandle loop) {
    if (threadIdx.x != 0) return;
    const long long n_req = c[0];
    unsigned int next = 0, tail = 0, go = 0;
    if (c[3] == 0u && n_req > 0) {
        if (n_req <= wave_tail) tail = static_cast<unsigned int>(n_req);
        else next = static_cast<unsigned int>(n_req);
    }
    if (next) {
        const unsigned int r = c[kWcRounds] + 1u;
        c[kWcRounds] = r;
        if (static_cast<long long>(r) >= max_rounds) c[kWcBound] = 1u;
        else go = 1u;
    }
    c[kWcNext] = next;
    c[kWcTail] = tail;
    cudaGraphSetConditional(loop, go);
}

cudaError_t launch_wave_decide(unsigned int* counters, long long wave_tail, long long max_rounds,
                               cudaGraphConditionalHandle loop, cudaStream_t stream) {
    k_wave_decide<<<1, 32, 0, stream>>>(counters, wave_tail, max_rounds, loop);
    return cudaGetLastError();
}

cudaError_t launch_newton(const DScene& S, const TraceArgs& A, const WaveArgs& W, long long n_req, cudaStream_t stream) {
    if (n_req <= 0) return cudaSuccess;
    if (S.max_nodes <= kGroup && W.group_newton) {
        const long long threads = n_req * kGroup;
        k_newton_grp<<<static_cast<unsigned>((threads + 127) / 128), 128, 0, stream>>>(S, A, W, n_req);
    } else if (S.max_nodes <= kGroup && W.newton_group_max > 0) {
        const long long threads = std::max(n_req, std::min(n_req, W.newton_group_max) * kGroup);
        k_newton_auto<<<static_cast<unsigned>((threads + 127) / 128), 128, 0, stream>>>(S, A, W, n_req);
    } else {
        k_newton<<<static_cast<unsigned>((n_req + 127) / 128), 128, 0, stream>>>(S, A, W, n_req);
    }
    return cudaGetLastError();
}

cudaError_t launch_resume(const DScene& S, const TraceArgs& A, const WaveArgs& W, const NewtonRequest* reqs,
                          const int* rays, long long n, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    k_resume<<<static_cast<unsigned>((n + 127) / 128), 128, 0, stream>>>(S, A, W, reqs, rays, n);
    return cudaGetLastError();
}

// Leaf records (DScene::leaf_rec) from the leaf order and the cull tables: one
// thread per leaf slot.
__global__ void k_leaf_records(DScene S, int n_slots, float4* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_slots) return;
    const int obj = S.leaf_objects[k], sub = S.obj_sub[obj];
    const bool patch = S.obj_kind[obj] == BBRT_OBJ_PATCH;
    float lo[3] = { -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F }, hi[3] = { CUDART_INF_F, CUDART_INF_F, CUDART_INF_F };
    const int nb = S.n_blocks_side * S.n_blocks_side;
    if (patch && S.c_block_box && nb > 0) {
        const float* b = S.c_block_box + 6LL * nb * sub;
        for (int a = 0; a < 3; ++a) { lo[a] = b[a]; hi[a] = b[3 + a]; }
        for (int j = 1; j < nb; ++j)
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], b[6 * j + a]);
                hi[a] = fmaxf(hi[a], b[6 * j + 3 + a]);
            }
    }
    out[2LL * k] = make_float4(lo[0], lo[1], lo[2], hi[0]);
    out[2LL * k + 1] = make_float4(hi[1], hi[2], __int_as_float(patch ? sub : ~sub), __int_as_float(obj));
}

// DScene::quad_box: a block of 256 threads per patch; thread m takes the cell
// with Morton index m, then the union of four children level by level.
__global__ void __launch_bounds__(256) k_quad_boxes(DScene S, float* __restrict__ out) {
    __shared__ float box[256][6];
    const int nc = S.coarse_n - 1, m = threadIdx.x;
    const float* cells = S.c_cell_box + 6LL * nc * nc * blockIdx.x;
    float* q = out + 6LL * kQuadNodes * blockIdx.x;
    int i = 0, j = 0;
    for (int b = 0; b < 4; ++b) {
        j |= (m >> (2 * b) & 1) << b;
        i |= (m >> (2 * b + 1) & 1) << b;
    }
    const bool in = i < nc && j < nc;
    for (int a = 0; a < 6; ++a) box[m][a] = in ? cells[6 * (i * nc + j) + a] : (a < 3 ? CUDART_INF_F : -CUDART_INF_F);
    int first = 84, count = 256;   // nodes of the level before, nodes of the level
    while (true) {
        if (m < count)
            for (int a = 0; a < 6; ++a) q[6 * (first + m) + a] = box[m][a];
        if (count == 4) break;
        __syncthreads();
        float u[6];
        count >>= 2;
        first -= count;
        if (m < count)
            for (int a = 0; a < 6; ++a) {
                u[a] = box[4 * m][a];
                for (int k = 1; k < 4; ++k) u[a] = a < 3 ? fminf(u[a], box[4 * m + k][a]) : fmaxf(u[a], box[4 * m + k][a]);
            }
        __syncthreads();
        if (m < count)
            for (int a = 0; a < 6; ++a) box[m][a] = u[a];
        __syncthreads();
    }
}

cudaError_t launch_quad_boxes(const DScene& S, int n_patches, float* out, cudaStream_t st) {
    if (n_patches <= 0) return cudaSuccess;
    k_quad_boxes<<<static_cast<unsigned>(n_patches), 256, 0, st>>>(S, out);
    return cudaGetLastError();
}

cudaError_t launch_leaf_records(const DScene& S, int n_slots, float4* out, cudaStream_t st) {
    if (n_slots <= 0) return cudaSuccess;
    k_leaf_records<<<static_cast<unsigned>((n_slots + 127) / 128), 128, 0, st>>>(S, n_slots, out);
    return cudaGetLastError();
}

// ---- BounceMapDriver::run on the device ------------------------------------

// Launch ray r = (point q, direction ti * phi_n + pj) of the sweep
// (BounceMapDriver.hpp:195-237): the point's frame (origin, t1, t2, n) and
// the direction tables come from the host; the expression and its rounding
// (no fused multiply-add in this file) are the reference's.
__global__ void k_bounce_rays(const double* __restrict__ frames, const double* __restrict__ trig, int theta_n,
                              int phi_n, long long n, double* __restrict__ org, double* __restrict__ dir) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= n) return;
    const long long dirs_per = static_cast<long long>(theta_n) * phi_n;
    const long long q = r / dirs_per, dk = r % dirs_per;
    const int ti = static_cast<int>(dk / phi_n), pj = static_cast<int>(dk % phi_n);
    const double* F = frames + 12 * q;
    const double m = trig[ti], st_ = trig[theta_n + ti], cp = trig[2 * theta_n + pj], sp = trig[2 * theta_n + phi_n + pj];
    org[3 * r] = F[0];
    org[3 * r + 1] = F[1];
    org[3 * r + 2] = F[2];
    dir[3 * r] = F[3] * st_ * cp + F[6] * st_ * sp + F[9] * m;
    dir[3 * r + 1] = F[4] * st_ * cp + F[7] * st_ * sp + F[10] * m;
    dir[3 * r + 2] = F[5] * st_ * cp + F[8] * st_ * sp + F[11] * m;
}

// Per grid point, by a warp: the largest bounce count over non-Error
// directions, the number of Error directions, and the first direction reaching
// the maximum (BounceMapDriver.hpp:199-240).  Lanes take directions 32 apart;
// the winner is the smallest direction with the largest count, as in the
// ordered loop.  (A thread per point left all but a few SMs idle and waited for
// two loads per direction one after the other: with 147 points of 960 directions
// 0.3 of a bounce map's 1.4 ms.)
__global__ void k_bounce_reduce(const int* __restrict__ status, const int* __restrict__ bounces, long long points,
                                int dirs_per, int* __restrict__ max_out, int* __restrict__ err_out,
                                int* __restrict__ best_out) {
    const long long q = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
    if (q >= points) return;   // whole warps
    const int lane = threadIdx.x & 31;
    int best = -1, nerr = 0, bdir = dirs_per;
    for (int k = lane; k < dirs_per; k += 32) {
        const long long r = q * dirs_per + k;
        const int s = status[r], b = bounces[r];
        if (s != BBRT_RAY_ESCAPED && s != BBRT_RAY_MAX_BOUNCES) ++nerr;
        else if (b > best) { best = b; bdir = k; }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int ob = __shfl_xor_sync(kFull, best, off), od = __shfl_xor_sync(kFull, bdir, off);
        nerr += __shfl_xor_sync(kFull, nerr, off);
        if (ob > best || (ob == best && od < bdir)) { best = ob; bdir = od; }
    }
    if (lane == 0) {
        max_out[q] = best < 0 ? 0 : best;
        err_out[q] = nerr;
        best_out[q] = best < 0 ? -1 : bdir;
    }
}

// PlaneSourceDriver's rays (PlaneSourceDriver.hpp:190-243): source (i, j) of the
// nx x ny grid from the host's coordinate tables (`grid`: nx values along axis
// aa, then ny along ab), one direction.
__global__ void k_plane_rays(const double* __restrict__ grid, int nx, int ny, int aa, int ab, int ac, double c, double dx,
                             double dy, double dz, double* __restrict__ org, double* __restrict__ dir) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= static_cast<long long>(nx) * ny) return;
    const long long i = r / ny;
    org[3 * r + aa] = grid[i];
    org[3 * r + ab] = grid[nx + (r - i * ny)];
    org[3 * r + ac] = c;
    dir[3 * r] = dx;
    dir[3 * r + 1] = dy;
    dir[3 * r + 2] = dz;
}

cudaError_t launch_plane_rays(const double* grid, int nx, int ny, int aa, int ab, int ac, double c, const double d[3],
                              double* org, double* dir, cudaStream_t st) {
    const long long n = static_cast<long long>(nx) * ny;
    k_plane_rays<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(grid, nx, ny, aa, ab, ac, c, d[0], d[1], d[2], org, dir);
    return cudaGetLastError();
}

cudaError_t launch_bounce_rays(const double* frames, const double* trig, int theta_n, int phi_n, long long n,
                               double* org, double* dir, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_bounce_rays<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(frames, trig, theta_n, phi_n, n, org, dir);
    return cudaGetLastError();
}

cudaError_t launch_bounce_reduce(const int* status, const int* bounces, long long points, int dirs_per, int* max_out,
                                 int* err_out, int* best_out, cudaStream_t st) {
    if (points <= 0) return cudaSuccess;
    k_bounce_reduce<<<static_cast<unsigned>((points + 3) / 4), 128, 0, st>>>(status, bounces, points, dirs_per,
                                                                              max_out, err_out, best_out);
    return cudaGetLastError();
}

// Check of the FP32 node test (bbrt_node_test_check): ray i against box i
// with bound t best[i]: out[2i] = ray_box_exact, out[2i + 1] = node_box_f32
// (-2 when the ray's FP32 values are outside the bound's range).
__global__ void k_node_check(DScene S, const double* __restrict__ o, const double* __restrict__ d,
                             const double* __restrict__ best, long long n, const double* __restrict__ boxes,
                             int* __restrict__ out) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const V3 oo = load3(o + 3 * i), dd = load3(d + 3 * i);
    const double inv[3] = { 1.0 / dd.x, 1.0 / dd.y, 1.0 / dd.z };
    out[2 * i] = ray_box_exact(oo, inv, boxes + 6 * i, best[i]) ? 1 : 0;
    const CullRay c = make_cull_ray(S, -1, oo, dd);
    NodeRay nr;
    __align__(8) float b32[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) b32[k] = static_cast<float>(boxes[6 * i + k]);
    const bool ok = finite3(oo) && finite3(dd) && make_node_ray(S, c, nr);
    nr.set_best(best[i]);
    out[2 * i + 1] = ok ? node_box_f32(b32, nr) : -2;
}

cudaError_t launch_node_check(const DScene& S, const double* o, const double* d, const double* best, long long n,
                              const double* boxes, int* out, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    k_node_check<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(S, o, d, best, n, boxes, out);
    return cudaGetLastError();
}

cudaError_t launch_query(const DScene& S, const QueryArgs& Q, cudaStream_t stream) {
    if (Q.n <= 0) return cudaSuccess;
    const unsigned blocks = static_cast<unsigned>((Q.n + 127) / 128);
    if (Q.mode != BBRT_QUERY_BVH) k_query<<<blocks, 128, 0, stream>>>(S, Q);
    else if (S.max_nodes > 0) k_query_bvh<true><<<blocks, 128, 0, stream>>>(S, Q);
    else k_query_bvh<false><<<blocks, 128, 0, stream>>>(S, Q);
    return cudaGetLastError();
}

}  // namespace bbrt
