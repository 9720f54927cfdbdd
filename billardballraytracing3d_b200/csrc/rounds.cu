// A round of the wavefront trace as two kernels: k_walk (tree) and k_stage1
// (patches), with k_newton after them.
//
// k_walk, a thread per ray, takes the last round's Newton result, finishes the
// query (bounce, escape, error, or another solve of it), and walks the tree
// for the next query with no bound on t, which lists the leaves whose box the
// ray meets in the reference's visiting order.  k_stage1, a warp per sixteen
// rays, runs the patches of those leaves: their boxes, then block boxes, cell
// boxes and triangles as compacted work lists over all of the warp's rays, and
// keeps each ray's stage-1 hits in visiting order.  The first becomes a Newton
// request; the others are taken up by k_walk, each leaf's box tested again with
// the best t found before it.  (Which leaves the reference visits, and why that
// test decides it: see ray_warp.cu.)
//
// What this is for: one kernel that walks and runs stage 1 (advance.cu) holds
// 128 registers a thread for the FP64 triangle tests, 16 warps on an SM, and
// spends its time on the latency of both; apart, the walk is a short loop at
// twice the warps and a warp's stage-1 lists are full.  About half more
// patches are tested than a walk that stops at the first hit would test.
//
// Rays with more leaves or hits than their lists hold, and rays that cannot be
// culled, go to the overflow list and are finished a warp per ray.
//
// Compiled with -fmad=false like the rest of the trace path (see exact.cuh).
//
// Reference (manuelarturosantana/BillardBallRayTracing3D):
//   RayTracingDriver::trace_ray   include/RayTracingDriver.hpp:172-242
//   BVH::intersect                include/BVH.hpp:75-128
//   SurfacePatch::intersect       include/ScatObjects/SurfacePatch.hpp:253-303
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>

#include "trace_common.cuh"

namespace bbrt {
namespace {

constexpr int kWalkThreads = 256;

__device__ __forceinline__ double* res_of(const WaveArgs& W, int i, int e) {
    return W.res_data + (static_cast<long long>(i) * kSplitResults + e) * kResData;
}

// Ends a single query: its record is all it writes (finish_ray then has nothing
// to write).
__device__ __forceinline__ void end_query(const TraceArgs& A, int i, RayCtx& r, const QHit& h) {
    write_hit(static_cast<bbrt_hit*>(A.query_out) + i, h);
    r.status = BBRT_RAY_ESCAPED;
}

// FP64 node test of ray i from its saved state.
__device__ __forceinline__ bool saved_box_exact(const WaveArgs& W, int i, const double* box, double best_t) {
    const V3 o = load3(W.o + 3LL * i), d = load3(W.d + 3LL * i);
    const double inv[3] = { 1.0 / d.x, 1.0 / d.y, 1.0 / d.z };
    return ray_box_exact(o, inv, box, best_t);
}

// The leaves ray i meets, in visiting order, into W.leaves; their number, or -1
// when there are more than the list holds.
template <bool STATS>
__device__ __forceinline__ int list_leaves(const DScene& S, const WaveArgs& W, int i, int member, const V3& d,
                                           const CullRay& cr, CountersT<STATS>& ctr) {
    NodeRay nr;
    const bool f32 = make_node_ray(S, cr, nr);
    // 1/d_a < 0 (finite d): the reference's child order
    const unsigned neg = (__double2hiint(d.x) < 0 ? 1u : 0u) | (__double2hiint(d.y) < 0 ? 2u : 0u) |
                         (__double2hiint(d.z) < 0 ? 4u : 0u);
    int* out = W.leaves + static_cast<long long>(i) * kSplitLeaves;
    int stack[32];
    int sp = 0, n = 0;
    const int root = root_node(S, member);
    int ref = S.m_ref[member < 0 ? 0 : member];
    int dec = f32 ? node_box_f32(S.node_box32 + 6LL * root, nr) : -1;
    ++ctr.node_tests;
    if (dec < 0) dec = saved_box_exact(W, i, S.node_box + 6LL * root, CUDART_INF);
    if (!dec) return 0;
    while (true) {
        if (ref >= 0) {
            const float4* rec = S.pair_rec + 4LL * ref;
            const float4 a = rec[0], b = rec[1], c = rec[2], v = rec[3];
            int l = -1, r = -1;
            ctr.node_tests += 2;
            if (f32) {
                l = node_box_f32(a.x, a.y, a.z, a.w, b.x, b.y, nr);
                r = node_box_f32(b.z, b.w, c.x, c.y, c.z, c.w, nr);
            }
            if ((l | r) < 0) {
                const double* box = S.node_box + 6LL * __float_as_int(v.x);
                if (f32) ctr.node_f64 += (l < 0 ? 1 : 0) + (r < 0 ? 1 : 0);
                if (l < 0) l = saved_box_exact(W, i, box, CUDART_INF);
                if (r < 0) r = saved_box_exact(W, i, box + 6, CUDART_INF);
            }
            const bool right_first = (neg >> __float_as_int(v.w)) & 1u;
            const int lref = __float_as_int(v.y), rref = __float_as_int(v.z);
            if (l && r) {
                ref = right_first ? rref : lref;
                stack[sp++] = right_first ? lref : rref;   // depth of a median-split tree: at most 25
                continue;
            }
            if (l || r) {
                ref = l ? lref : rref;
                continue;
            }
        } else {
            if (n == kSplitLeaves) return -1;
            out[n++] = ~ref;
        }
        if (sp == 0) return n;
        ref = stack[--sp];
    }
}

// One thread per runnable ray.  Bound by the latency of dependent node records
// (64 bytes, L1), so the point is warps: 64 registers, 32 warps on an SM.
template <bool STATS>
__global__ void __launch_bounds__(kWalkThreads, 4) k_walk(DScene S, TraceArgs A, WaveArgs W) {
    const long long n = W.count_dev ? static_cast<long long>(*W.count_dev) : W.n_runnable;
    const int lane = threadIdx.x & 31;
    const long long t_start = clock64();
    CountersT<STATS> ctr;
    RayTallyT<STATS> tally;
    for (long long base = static_cast<long long>(blockIdx.x) * kWalkThreads; base < n;
         base += static_cast<long long>(gridDim.x) * kWalkThreads) {
        const long long j = base + threadIdx.x;
        NewtonRequest rq;
        bool ask = false, listed = false, over = false;
        int i = -1;
        if (j < n) {
            RayCtx r;
            bool query = false;
            CountersT<STATS> cray;
            if (W.runnable == nullptr) {
                i = W.order ? W.order[j] : static_cast<int>(j);
                if (A.query_out) {
                    r = start_query(A, i);
                } else {
                    init_outputs(A, i);
                    r = start_ray(A, i);
                }
                if (r.status < 0) {
                    if (A.max_bounces > 0) query = true;
                    else r.status = BBRT_RAY_MAX_BOUNCES;
                }
            } else {
                const NewtonRequest done = W.runnable[j];
                i = done.ray;
                r.member = A.ray_member ? A.ray_member[i] : -1;
                r.o = load3(W.o + 3LL * i);
                r.d = load3(W.d + 3LL * i);
                r.bounces = W.bounces[i];
                r.status = -1;
                r.err_obj = -1;
                r.ev0 = r.ev1 = 0.0;
                const int e = done.entry & 1, k = done.entry >> 1;
                const SplitHit* hits = W.hits + static_cast<long long>(i) * kSplitHits;
                QHit h;
                h.err = W.res_err[static_cast<long long>(i) * kSplitResults + e];
                h.obj = done.obj;
                int best = -1;   // hit << 1 | result slot
                if (!h.err) {
                    best = W.best[i];
                    double best_t = best < 0 ? CUDART_INF : *res_of(W, i, best & 1);
                    const double t = *res_of(W, i, e);
                    if (t < best_t) {
                        best_t = t;
                        best = k << 1 | e;
                    }
                    // the query's later hits, in leaves not pruned by best_t
                    const int n_hits = W.n_hits[i];
                    for (int m = k + 1; m < n_hits && !ask; ++m) {
                        const SplitHit c = hits[m];
                        if (c.leaf != hits[k].leaf && best_t < CUDART_INF &&
                            !saved_box_exact(W, i, S.leaf_box + 6LL * c.leaf, best_t))
                            continue;
                        rq.ray = i;
                        rq.entry = m << 1 | (best >= 0 && (best & 1) == 0 ? 1 : 0);
                        rq.obj = c.obj;
                        rq.key = c.key;
                        rq.t0 = c.t;
                        W.best[i] = best;
                        ask = true;
                    }
                    if (!ask) h.obj = best < 0 ? -1 : hits[best >> 1].obj;
                }
                if (!ask) {
                    if (h.err || h.obj >= 0) {
                        const double* rd = res_of(W, i, h.err ? e : best & 1);
                        h.t = rd[0];
                        h.p = v3(rd[1], rd[2], rd[3]);
                        h.n = v3(rd[4], rd[5], rd[6]);
                        h.u = rd[7];
                        h.v = rd[8];
                        h.ev0 = rd[9];
                        h.ev1 = rd[10];
                    }
                    ++tally.queries;
                    if (A.query_out) {
                        end_query(A, i, r, h);
                    } else if (step_ray(S, A, i, r, h)) {
                        if (r.bounces < A.max_bounces) query = true;
                        else r.status = BBRT_RAY_MAX_BOUNCES;
                    }
                }
            }
            if (query) {
                double* so = W.o + 3LL * i;
                double* sd = W.d + 3LL * i;
                so[0] = r.o.x; so[1] = r.o.y; so[2] = r.o.z;
                sd[0] = r.d.x; sd[1] = r.d.y; sd[2] = r.d.z;
                W.bounces[i] = r.bounces;
                if (!cull_ok(S, r.member, A.cull, r.o, r.d)) {
                    over = true;
                } else {
                    const CullRay cr = make_cull_ray(S, r.member, r.o, r.d);
                    const int found = list_leaves<STATS>(S, W, i, r.member, r.d, cr, cray);
                    if (found < 0) {
                        over = true;
                    } else if (found == 0) {
                        ++tally.queries;
                        r.o = load3(W.o + 3LL * i);
                        r.d = load3(W.d + 3LL * i);
                        QHit h;
                        h.err = 0;
                        h.obj = -1;
                        if (A.query_out) end_query(A, i, r, h);
                        else step_ray(S, A, i, r, h);
                    } else {
                        W.n_leaves[i] = found;
                        listed = true;
                    }
                }
            }
            if (!ask && r.status >= 0) {
                finish_ray(A, i, r);
                tally.bounces += r.bounces;
                tally.hist[r.status]++;
            }
            if constexpr (STATS) {
                add_ray_work(A, i, cray);
                ctr.node_tests += cray.node_tests;
                ctr.node_f64 += cray.node_f64;
            }
        }
        __syncwarp();
        // requests, overflows and rays with leaves: three lists, one round trip
        const unsigned m_ask = __ballot_sync(kFull, ask), m_over = __ballot_sync(kFull, over),
                       m_list = __ballot_sync(kFull, listed);
        unsigned at = 0;
        if (lane < 3) {
            const int add = __popc(lane == 0 ? m_ask : lane == 1 ? m_over : m_list);
            if (add) at = atomicAdd(&W.counters[lane], static_cast<unsigned>(add));
        }
        const unsigned before = (1u << lane) - 1u;
        const unsigned a_ask = __shfl_sync(kFull, at, 0), a_over = __shfl_sync(kFull, at, 1), a_list = __shfl_sync(kFull, at, 2);
        if (ask) W.req[a_ask + __popc(m_ask & before)] = rq;
        if (over) W.overflow[a_over + __popc(m_over & before)] = i;
        if (listed) W.listed[a_list + __popc(m_list & before)] = i;
        // a launch that runs far past any real round gives up (see advance.cu)
        if (clock64() - t_start > W.watchdog_cycles) {
            atomicOr(&W.counters[3], 1u);
            break;
        }
    }
    __syncwarp();
    flush_stats(A, ctr, tally);
}

// ---- stage 1 -----------------------------------------------------------------

constexpr int kRays = 16;           // rays of a warp
constexpr int kS1Warps = 4;         // warps per block
constexpr int kMaxCand = 32 * kSplitLeafSlots + 32;
constexpr int kBlockUnroll = 2, kCellUnroll = 1;   // box loads in flight per lane (4 and 2: more spills, 1 % slower)
constexpr int kBlkSmall = 512;      // blocks of a batch of 32 patches of 16 each
constexpr int kBlkCap = kBlkSmall / 2;   // other grids: 4 bytes an entry, tested when full
constexpr int kCellCap = 128;

// One warp's shared memory.
struct __align__(16) S1Work {
    float4 cr_a[kRays], cr_b[kRays];           // cull rays: origin, inflation; 1 / direction
    double od[6][kRays];                       // origins, directions
    int ray[kRays], n_hits[kRays], leaf0[kRays];
    unsigned char leaf_ray[kRays * kSplitLeaves];   // the leaves in (ray, visiting) order: their rays
    int sub[kMaxCand], slot[kMaxCand];         // candidates in that order: patch or ~triangle, slot
    unsigned char cand_ray[kMaxCand], cand_pos[kMaxCand];   // ... ray, place of its leaf
    union {                                    // passing blocks of a batch
        unsigned short small[kBlkSmall];       // candidate << 8 | row << 4 | column
        int any[kBlkCap];                      // candidate << 24 | block
    } blk;
    int cell[kCellCap];                        // passing cells: candidate of the batch << 24 | cell
    int cells[kRays], tris[kRays];             // box and triangle tests (statistics)
};

__device__ __forceinline__ CullRay s1_cull(const S1Work& w, int r) {
    const float4 a = w.cr_a[r], b = w.cr_b[r];
    CullRay c;
    c.ox = a.x; c.oy = a.y; c.oz = a.z; c.delta = a.w;
    c.ix = b.x; c.iy = b.y; c.iz = b.z;
    return c;
}

// Triangle tests of the n cells waiting, 32 at a time; a hit goes to the lane of
// its candidate, which keeps the (t, key) minimum.
__device__ __forceinline__ void s1_tris(const DScene& S, S1Work& w, int c0, int n_cells, int lane, Stage1& mine) {
    const int n = S.coarse_n, nc = n - 1, total = 6 * n_cells;
    for (int p0 = 0; p0 < total; p0 += 32) {
        const int p = p0 + lane;
        Stage1 s;
        int owner = 0;
        if (p < total) {
            const int ce = p / 6, e = w.cell[ce], cl = e & 0xFFFFFF, i = cl / nc;
            owner = e >> 24;
            const int sub = w.sub[c0 + owner], r = w.cand_ray[c0 + owner];
            stage1_tri(S.c_xyz + static_cast<long long>(sub) * n * n * 3, S.c_cell + static_cast<long long>(sub) * nc * nc * 4,
                       n, i, cl - i * nc, p - 6 * ce, v3(w.od[0][r], w.od[1][r], w.od[2][r]),
                       v3(w.od[3][r], w.od[4][r], w.od[5][r]), s);
        }
        for (unsigned hits = __ballot_sync(kFull, s.have); hits; hits &= hits - 1) {
            const int src = __ffs(hits) - 1;
            const double t = __shfl_sync(kFull, s.t, src);
            const int key = __shfl_sync(kFull, s.key, src);
            const int to = __shfl_sync(kFull, owner, src);
            if (lane == to) mine.consider(t, key);
        }
    }
}

// Stage 1 of the P <= 32 candidates from c0 on: lane c returns candidate c's
// winner.  Patches of at most 4 x 4 blocks of 4 x 4 cells: sixteen lanes take a
// patch's blocks, then a block's cells, several at a time so that their loads
// are in flight together.
template <bool STATS>
__device__ __forceinline__ Stage1 s1_batch_small(const DScene& S, S1Work& w, int c0, int P, int lane) {
    const int nc = S.coarse_n - 1, NB = S.n_blocks_side, NB2 = NB * NB;
    const unsigned lt = (1u << lane) - 1u;
    const int half = lane >> 4, hl = lane & 15;
    const int hi = hl / NB, hj = hl - hi * NB;
    Stage1 mine;
    int n_blk = 0;
    constexpr int U = kBlockUnroll, V = kCellUnroll;
    for (int p = 0; p < P; p += 2 * U) {
        int ray[U];
        float2 b[U][3];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int c = p + 2 * k + half;
            ray[k] = -1;
            if (c < P && hl < NB2) {
                const int sub = w.sub[c0 + c];
                if (sub >= 0) {
                    ray[k] = w.cand_ray[c0 + c];
                    const float2* src = reinterpret_cast<const float2*>(S.c_block_box + (static_cast<long long>(sub) * NB2 + hl) * 6);
#pragma unroll
                    for (int a = 0; a < 3; ++a) b[k][a] = src[a];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (STATS && ray[k] >= 0) atomicAdd(&w.cells[ray[k]], 1);
            const bool pass = ray[k] >= 0 && cull_box(b[k][0], b[k][1], b[k][2], s1_cull(w, ray[k]));
            const unsigned m = __ballot_sync(kFull, pass);
            if (pass) w.blk.small[n_blk + __popc(m & lt)] = static_cast<unsigned short>((p + 2 * k + half) << 8 | hi << 4 | hj);
            n_blk += __popc(m);
        }
    }
    __syncwarp();
    int n_cell = 0;
    for (int p = 0; p < n_blk; p += 2 * V) {
        int entry[V];   // candidate << 24 | cell, or -1
        float2 b[V][3];
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const int c = p + 2 * k + half;
            entry[k] = -1;
            if (c < n_blk) {
                const int e = w.blk.small[c], i = ((e >> 4) & 15) * 4 + (hl >> 2), j = (e & 15) * 4 + (hl & 3);
                if (i < nc && j < nc) {
                    const int cell = i * nc + j;
                    entry[k] = (e >> 8) << 24 | cell;
                    const float2* src = reinterpret_cast<const float2*>(
                        S.c_cell_box + (static_cast<long long>(w.sub[c0 + (e >> 8)]) * nc * nc + cell) * 6);
#pragma unroll
                    for (int a = 0; a < 3; ++a) b[k][a] = src[a];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < V; ++k) {
            bool pass = entry[k] >= 0;
            if (pass) {
                const int r = w.cand_ray[c0 + (entry[k] >> 24)];
                if (STATS) atomicAdd(&w.cells[r], 1);
                pass = cull_box(b[k][0], b[k][1], b[k][2], s1_cull(w, r));
                if (STATS && pass) atomicAdd(&w.tris[r], 6);
            }
            const unsigned m = __ballot_sync(kFull, pass);
            if (pass) w.cell[n_cell + __popc(m & lt)] = entry[k];
            n_cell += __popc(m);
        }
        if (n_cell > kCellCap - 32 * V || p + 2 * V >= n_blk) {
            __syncwarp();
            s1_tris(S, w, c0, n_cell, lane, mine);
            __syncwarp();
            n_cell = 0;
        }
    }
    return mine;
}

// The same for any grid: blocks and cells flattened over the batch.
template <bool STATS>
__device__ __forceinline__ Stage1 s1_batch(const DScene& S, S1Work& w, int c0, int P, int lane) {
    const int nc = S.coarse_n - 1, B = S.block_cells, B2 = B * B, NB = S.n_blocks_side, NB2 = NB * NB;
    const unsigned lt = (1u << lane) - 1u;
    Stage1 mine;
    int n_blk = 0, n_cell = 0;
    const int blocks = P * NB2;
    for (int b0 = 0; b0 < blocks; b0 += 32) {
        const int x = b0 + lane, c = x / NB2, b = x - c * NB2;
        bool pass = x < blocks;
        if (pass) {
            const int sub = w.sub[c0 + c], r = w.cand_ray[c0 + c];
            pass = sub >= 0;
            if (STATS && pass) atomicAdd(&w.cells[r], 1);
            if (pass) pass = cull_box(S.c_block_box + (static_cast<long long>(sub) * NB2 + b) * 6, s1_cull(w, r));
        }
        const unsigned m = __ballot_sync(kFull, pass);
        if (pass) w.blk.any[n_blk + __popc(m & lt)] = c << 24 | b;
        n_blk += __popc(m);
        if (b0 + 32 < blocks && n_blk <= kBlkCap - 32) continue;
        __syncwarp();
        const int cells = n_blk * B2;
        for (int y0 = 0; y0 < cells; y0 += 32) {
            const int y = y0 + lane, q = y / B2, k = y - q * B2;
            bool ok = y < cells;
            int cand = 0, cell = 0;
            if (ok) {
                const int e = w.blk.any[q], bb = e & 0xFFFFFF, bi = bb / NB, ki = k / B;
                const int i = bi * B + ki, j = (bb - bi * NB) * B + (k - ki * B);
                cand = e >> 24;
                cell = i * nc + j;
                ok = i < nc && j < nc;
            }
            if (ok) {
                const int r = w.cand_ray[c0 + cand];
                if (STATS) atomicAdd(&w.cells[r], 1);
                ok = cull_box(S.c_cell_box + (static_cast<long long>(w.sub[c0 + cand]) * nc * nc + cell) * 6, s1_cull(w, r));
                if (STATS && ok) atomicAdd(&w.tris[r], 6);
            }
            const unsigned cm = __ballot_sync(kFull, ok);
            if (ok) w.cell[n_cell + __popc(cm & lt)] = cand << 24 | cell;
            n_cell += __popc(cm);
            if (n_cell > kCellCap - 32) {
                __syncwarp();
                s1_tris(S, w, c0, n_cell, lane, mine);
                __syncwarp();
                n_cell = 0;
            }
        }
        n_blk = 0;
        __syncwarp();
    }
    s1_tris(S, w, c0, n_cell, lane, mine);
    __syncwarp();
    return mine;
}

// The round control of a graph-launched trace: no requests, or a watchdog stop:
// the rounds end.  At most wave_tail requests: the rounds end and the tail
// finishes those rays.  Otherwise the requests go to Newton and become the next
// round's runnable set; the loop repeats unless this was round max_rounds
// (flagged for the host as an error), so it ends whatever the counts.
__device__ void decide_round(unsigned int* c, const RoundControl& R) {
    volatile unsigned int* v = c;
    const long long n_req = v[0];
    unsigned int next = 0, tail = 0, go = 0;
    if (v[3] == 0u && n_req > 0) {
        if (n_req <= R.wave_tail) tail = static_cast<unsigned int>(n_req);
        else next = static_cast<unsigned int>(n_req);
    }
    if (next) {
        const unsigned int r = v[kWcRounds] + 1u;
        v[kWcRounds] = r;
        if (static_cast<long long>(r) >= R.max_rounds) v[kWcBound] = 1u;
        else go = 1u;
    }
    v[kWcNext] = next;
    v[kWcTail] = tail;
    cudaGraphSetConditional(R.loop, go);
}

// A warp per up to sixteen rays of W.listed (fewer in a round with fewer rays
// than the grid's warps can take sixteen of, a power of two that covers it).
template <bool SMALL, bool STATS>
__global__ void __launch_bounds__(kS1Warps * 32, 6) k_stage1(DScene S, TraceArgs A, WaveArgs W, RoundControl R) {
    extern __shared__ __align__(16) unsigned char s1_smem[];
    S1Work& w = reinterpret_cast<S1Work*>(s1_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const long long n = W.counters[2];
    const long long warps = static_cast<long long>(gridDim.x) * kS1Warps;
    const long long t_start = clock64();
    CountersT<STATS> ctr;
    RayTallyT<STATS> tally;
    int per = kRays;
    while (per > 1 && per / 2 * warps >= n) per >>= 1;
    while (true) {
        // groups are handed out one at a time: a warp's share of the patches varies
        unsigned int first_ray = 0;
        if (lane == 0) first_ray = atomicAdd(&W.counters[kWcGroup], static_cast<unsigned>(per));
        const long long g = __shfl_sync(kFull, first_ray, 0);
        if (g >= n) break;
        const int rays = static_cast<int>(min(static_cast<long long>(per), n - g));
        // ---- the rays and the list of their leaves
        int i = -1, count = 0;
        if (lane < rays) {
            i = W.listed[g + lane];
            count = W.n_leaves[i];
            const V3 o = load3(W.o + 3LL * i), d = load3(W.d + 3LL * i);
            const CullRay cr = make_cull_ray(S, A.ray_member ? A.ray_member[i] : -1, o, d);
            w.cr_a[lane] = make_float4(cr.ox, cr.oy, cr.oz, cr.delta);
            w.cr_b[lane] = make_float4(cr.ix, cr.iy, cr.iz, 0.0f);
            w.od[0][lane] = o.x; w.od[1][lane] = o.y; w.od[2][lane] = o.z;
            w.od[3][lane] = d.x; w.od[4][lane] = d.y; w.od[5][lane] = d.z;
            w.ray[lane] = i;
            w.n_hits[lane] = 0;
            if (STATS) w.cells[lane] = w.tris[lane] = 0;
        }
        int x = count;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFull, x, off);
            if (lane >= off) x += y;
        }
        const int n_leaf = __shfl_sync(kFull, x, 31);
        if (lane < rays) w.leaf0[lane] = x - count;
        for (int k = 0; k < count; ++k) w.leaf_ray[x - count + k] = static_cast<unsigned char>(lane);
        __syncwarp();
        // ---- a leaf per lane: its patches whose box the ray meets (triangles: all),
        // then stage 1, 32 of them at a time
        int n_cand = 0;
        for (int l0 = 0; l0 < n_leaf; l0 += 32) {
            int r = 0, first = 0, pos = 0;
            unsigned pass = 0;
            if (l0 + lane < n_leaf) {
                r = w.leaf_ray[l0 + lane];
                pos = l0 + lane - w.leaf0[r];
                const int leaf = W.leaves[static_cast<long long>(w.ray[r]) * kSplitLeaves + pos];
                const float4 b = S.leaf_node[2LL * leaf + 1];
                first = __float_as_int(b.z);
                const int slots = __float_as_int(b.w);
                const CullRay cr = s1_cull(w, r);
                for (int k = 0; k < slots; ++k) {
                    const LeafRec rec = load_leaf(S, first + k);
                    if (rec.sub() < 0 || cull_leaf(rec, cr)) pass |= 1u << k;
                    if (STATS && rec.sub() >= 0) {
                        atomicAdd(&w.cells[r], 1);
                        ++ctr.patch_tests;
                    }
                }
            }
            int y = __popc(pass);
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int z = __shfl_up_sync(kFull, y, off);
                if (lane >= off) y += z;
            }
            int at = n_cand + y - __popc(pass);
            for (unsigned m = pass; m; m &= m - 1, ++at) {
                const int slot = first + __ffs(m) - 1;
                w.sub[at] = __float_as_int(S.leaf_rec[2LL * slot + 1].z);
                w.slot[at] = slot;
                w.cand_ray[at] = static_cast<unsigned char>(r);
                w.cand_pos[at] = static_cast<unsigned char>(pos);
            }
            n_cand += __shfl_sync(kFull, y, 31);
            __syncwarp();
            const bool last = l0 + 32 >= n_leaf;
            int c0 = 0;
            for (; c0 < n_cand && (last || c0 + 32 <= n_cand); c0 += 32) {
                const int P = min(32, n_cand - c0);
                Stage1 s = SMALL ? s1_batch_small<STATS>(S, w, c0, P, lane) : s1_batch<STATS>(S, w, c0, P, lane);
                if (lane < P && w.sub[c0 + lane] < 0) {
                    const int q = w.cand_ray[c0 + lane];
                    QHit h;
                    CountersT<false> dummy;
                    s.have = triangle_intersect(S, ~w.sub[c0 + lane], v3(w.od[0][q], w.od[1][q], w.od[2][q]),
                                                v3(w.od[3][q], w.od[4][q], w.od[5][q]), h, dummy) != 0;
                    s.t = h.t;
                    s.key = 0;
                    ctr.tri_tests += 1;
                }
                // hits in visiting order
                const bool hit = lane < P && s.have;
                const unsigned hm = __ballot_sync(kFull, hit);
                if (hit) {
                    const int c = c0 + lane, q = w.cand_ray[c];
                    const unsigned peers = __match_any_sync(hm, q);
                    const int old = w.n_hits[q], place = old + __popc(peers & lt);
                    if (place < kSplitHits) {
                        SplitHit* out = W.hits + static_cast<long long>(w.ray[q]) * kSplitHits + place;
                        out->t = s.t;
                        out->obj = __float_as_int(S.leaf_rec[2LL * w.slot[c] + 1].w);
                        out->leaf = W.leaves[static_cast<long long>(w.ray[q]) * kSplitLeaves + w.cand_pos[c]];
                        out->key = s.key;
                    }
                    __syncwarp(hm);
                    if (lane == __ffs(peers) - 1) w.n_hits[q] = old + __popc(peers);
                }
                __syncwarp();
            }
            // fewer than 32 left: they go to the front and wait for the next leaves
            if (!last && c0 > 0) {
                const int k = c0 + lane;
                const bool keep = k < n_cand;
                const int sub = keep ? w.sub[k] : 0, slot = keep ? w.slot[k] : 0;
                const unsigned char cr = keep ? w.cand_ray[k] : 0, cp = keep ? w.cand_pos[k] : 0;
                __syncwarp();
                if (keep) {
                    w.sub[lane] = sub;
                    w.slot[lane] = slot;
                    w.cand_ray[lane] = cr;
                    w.cand_pos[lane] = cp;
                }
                n_cand -= c0;
                __syncwarp();
            }
        }
        // ---- each ray's first hit is its Newton request; none: it escapes
        bool ask = false, over = false;
        NewtonRequest rq;
        if (lane < rays) {
            const int hits = w.n_hits[lane];
            if (hits == 0) {
                RayCtx r;
                r.member = A.ray_member ? A.ray_member[i] : -1;
                r.o = v3(w.od[0][lane], w.od[1][lane], w.od[2][lane]);
                r.d = v3(w.od[3][lane], w.od[4][lane], w.od[5][lane]);
                r.bounces = W.bounces[i];
                r.err_obj = -1;
                r.ev0 = r.ev1 = 0.0;
                QHit h;
                h.err = 0;
                h.obj = -1;
                ++tally.queries;
                if (A.query_out) end_query(A, i, r, h);
                else step_ray(S, A, i, r, h);
                finish_ray(A, i, r);
                tally.bounces += r.bounces;
                tally.hist[r.status]++;
            } else if (hits > kSplitHits) {
                over = true;
            } else {
                const SplitHit c = W.hits[static_cast<long long>(i) * kSplitHits];
                W.n_hits[i] = hits;
                W.best[i] = -1;
                rq.ray = i;
                rq.entry = 0;
                rq.obj = c.obj;
                rq.key = c.key;
                rq.t0 = c.t;
                ask = true;
            }
            if constexpr (STATS) {
                CountersT<STATS> c;
                c.cell_tests = w.cells[lane];
                c.tri_tests = w.tris[lane];
                add_ray_work(A, i, c);
                ctr.cell_tests += c.cell_tests;
                ctr.tri_tests += c.tri_tests;
            }
        }
        const unsigned m_ask = __ballot_sync(kFull, ask), m_over = __ballot_sync(kFull, over);
        unsigned at = 0;
        if (lane < 2) {
            const int add = __popc(lane == 0 ? m_ask : m_over);
            if (add) at = atomicAdd(&W.counters[lane], static_cast<unsigned>(add));
        }
        const unsigned a_ask = __shfl_sync(kFull, at, 0), a_over = __shfl_sync(kFull, at, 1);
        if (ask) W.req[a_ask + __popc(m_ask & lt)] = rq;
        if (over) W.overflow[a_over + __popc(m_over & lt)] = i;
        if (__any_sync(kFull, clock64() - t_start > W.watchdog_cycles)) {
            if (lane == 0) atomicOr(&W.counters[3], 1u);
            break;
        }
        __syncwarp();
    }
    flush_stats(A, ctr, tally);
    // the last block to get here resets the hand-out and decides the round
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&W.counters[kWcTicket], 1u) == gridDim.x - 1) {
            __threadfence();
            W.counters[kWcTicket] = 0;
            W.counters[kWcGroup] = 0;
            if (R.on) decide_round(W.counters, R);
        }
    }
}

template <bool SMALL, bool STATS>
cudaError_t launch_stage1(const DScene& S, const TraceArgs& A, const WaveArgs& W, const RoundControl& R, int sm_count,
                          cudaStream_t stream) {
    constexpr int smem = kS1Warps * sizeof(S1Work);
    cudaError_t e = cudaFuncSetAttribute(k_stage1<SMALL, STATS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage1<SMALL, STATS>, kS1Warps * 32, smem);
    if (e != cudaSuccess) return e;
    const long long blocks = std::min<long long>(static_cast<long long>(std::max(per_sm, 1)) * sm_count,
                                                 (W.n_runnable + kS1Warps - 1) / kS1Warps);
    k_stage1<SMALL, STATS><<<static_cast<unsigned>(blocks), kS1Warps * 32, smem, stream>>>(S, A, W, R);
    return cudaGetLastError();
}

template <bool STATS>
cudaError_t launch_walk(const DScene& S, const TraceArgs& A, const WaveArgs& W, int sm_count, cudaStream_t stream) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk<STATS>, kWalkThreads, 0);
    if (e != cudaSuccess) return e;
    // a few times the resident blocks, so that blocks whose rays walk far are
    // made up for by others
    const long long blocks = std::min<long long>(4LL * std::max(per_sm, 1) * sm_count,
                                                 (W.n_runnable + kWalkThreads - 1) / kWalkThreads);
    k_walk<STATS><<<static_cast<unsigned>(blocks), kWalkThreads, 0, stream>>>(S, A, W);
    return cudaGetLastError();
}

}  // namespace

// k_walk and k_stage1 of a round (W.n_runnable sizes the grids; W.count_dev, if
// set, has the count).  R.on: the last block decides the graph's next round.
cudaError_t launch_round(const DScene& S, const TraceArgs& A, const WaveArgs& W, const RoundControl& R, int sm_count,
                         cudaStream_t stream) {
    if (W.n_runnable <= 0) return cudaSuccess;
    const bool stats = A.stats || A.ray_work, small = S.block_cells == 4 && S.n_blocks_side <= 4;
    const cudaError_t e = stats ? launch_walk<true>(S, A, W, sm_count, stream) : launch_walk<false>(S, A, W, sm_count, stream);
    if (e != cudaSuccess) return e;
    if (stats) return small ? launch_stage1<true, true>(S, A, W, R, sm_count, stream) : launch_stage1<false, true>(S, A, W, R, sm_count, stream);
    return small ? launch_stage1<true, false>(S, A, W, R, sm_count, stream) : launch_stage1<false, false>(S, A, W, R, sm_count, stream);
}

size_t split_workspace_bytes(long long n) {
    return (sizeof(double) * 6 + sizeof(int) * 3 + sizeof(int) * kSplitLeaves + sizeof(SplitHit) * kSplitHits +
            sizeof(int) * kSplitResults + sizeof(double) * kSplitResults * kResData + 2 * sizeof(NewtonRequest) +
            3 * sizeof(int)) * n + 24 * 256;
}

// Carves the workspace of a split round for n rays out of `ws`.
void split_layout(void* ws, long long n, WaveArgs& W, NewtonRequest*& req_a, NewtonRequest*& req_b) {
    char* p = static_cast<char*>(ws);
    auto take = [&](size_t bytes) { char* q = p; p += (bytes + 255) & ~static_cast<size_t>(255); return q; };
    W.o = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    W.d = reinterpret_cast<double*>(take(sizeof(double) * 3 * n));
    W.bounces = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.nres = nullptr;
    W.leaves = reinterpret_cast<int*>(take(sizeof(int) * kSplitLeaves * n));
    W.n_leaves = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.hits = reinterpret_cast<SplitHit*>(take(sizeof(SplitHit) * kSplitHits * n));
    W.n_hits = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.best = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.listed = reinterpret_cast<int*>(take(sizeof(int) * n));
    W.res_err = reinterpret_cast<int*>(take(sizeof(int) * kSplitResults * n));
    W.res_data = reinterpret_cast<double*>(take(sizeof(double) * kSplitResults * kResData * n));
    W.results = kSplitResults;
    req_a = reinterpret_cast<NewtonRequest*>(take(sizeof(NewtonRequest) * n));
    req_b = reinterpret_cast<NewtonRequest*>(take(sizeof(NewtonRequest) * n));
    W.overflow = reinterpret_cast<int*>(take(sizeof(int) * n));
}

}  // namespace bbrt
