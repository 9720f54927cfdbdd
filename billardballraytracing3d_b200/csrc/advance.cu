// k_advance: a round of the wavefront trace.  Runnable rays advance until each
// needs a Newton solve, overflows its resolved list, or finishes.
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

// What a lane's ray is doing.  Everything from M_FINISH on leaves the working
// loop for the retire / fetch step.
enum AdvMode {
    M_TRAV = 0,      // walking the BVH
    M_LEAF = 1,      // at the slots of a leaf
    M_S1 = 2,        // at a patch whose stage 1 is to be run
    M_S1_DONE = 3,   // stage 1 of that patch finished
    M_RESOLVE = 4,   // query finished: bounce, escape or error
    M_FINISH = 5,    // ray finished, its results written
    M_SUSPEND = 6,   // waiting for a Newton solve
    M_OVERFLOW = 7,  // more solves than the resolved list holds
    M_IDLE = 8,      // lane has no ray
    M_DRAINED = 9    // no runnable ray left
};

constexpr int kBlkQueue = 512;    // 32 patches of at most 16 blocks
constexpr int kCellQueue = 128;   // cells waiting for their triangle tests
constexpr int kCellFlush = kCellQueue - 64;

// One warp's shared memory: its rays (lane's slot), and the work lists of a
// batch of stage 1s.
struct WarpWork {
    float4 cr_a[32];                   // cull ray: origin, inflation
    float4 cr_b[32];                   // 1 / direction, patch of the pending stage 1 (int bits)
    double od[6][32];                  // origin xyz, direction xyz
    unsigned short blk[kBlkQueue];     // passing blocks: lane << 8 | block row << 4 | block column
    unsigned short cell[kCellQueue];   // passing cells: lane << 8 | row << 4 | column
    unsigned char lane_of[32];         // lanes of the batch
    float e[32];                       // margin of the FP32 node test; negative: nodes tested in FP64
    int cells[32], tris[32];           // box and triangle tests of a lane's patch (statistics)
};
static_assert(sizeof(WarpWork) % 16 == 0, "per-warp blocks must keep 16-byte alignment");

__device__ __forceinline__ CullRay work_cull_ray(const WarpWork& w, int lane) {
    const float4 a = w.cr_a[lane], b = w.cr_b[lane];
    CullRay c;
    c.ox = a.x; c.oy = a.y; c.oz = a.z; c.delta = a.w;
    c.ix = b.x; c.iy = b.y; c.iz = b.z;
    return c;
}
__device__ __forceinline__ V3 work_o(const WarpWork& w, int lane) { return v3(w.od[0][lane], w.od[1][lane], w.od[2][lane]); }
__device__ __forceinline__ V3 work_d(const WarpWork& w, int lane) { return v3(w.od[3][lane], w.od[4][lane], w.od[5][lane]); }

constexpr int kNone = static_cast<int>(0x80000000u);

// Per-lane state of the query being walked.
struct AdvState {
    bool use_cull;
    unsigned neg;        // bit a: 1/d_a < 0 (the reference's child order)
    double best_t;
    int best_obj;        // -1: no hit yet
    int best_e;          // resolved entry of the best patch hit (or of the failed solve), -1 for a triangle
    int err;
    int ref;             // node to enter next, known to pass (a reference of DScene::pair_rec), or kNone
    int sp;
    int untested;        // stack entries below this were tested with a larger best_t, or not at all
    int slot, slot_end;  // leaf slots still to look at
    int obj;             // object of the pending stage 1
    Stage1 s1;
};

// bit a set: 1.0 / d_a < 0.0 (also for -0, whose inverse is -inf; not for
// -inf, whose inverse is -0, nor for NaN)
__device__ __forceinline__ unsigned neg_bit(double d) {
    return (__double2hiint(d) < 0 && d >= -1.7976931348623157e308) ? 1u : 0u;
}

__device__ __forceinline__ void adv_start_query(const DScene& S, const TraceArgs& A, const WaveArgs& W, int member,
                                                const V3& o, const V3& d, int lane, WarpWork& ww, AdvState& q,
                                                int* stack) {
    q.neg = neg_bit(d.x) | (neg_bit(d.y) << 1) | (neg_bit(d.z) << 2);
    q.use_cull = cull_ok(S, member, A.cull, o, d);
    const bool node32 = W.node_f32 && finite3(o) && finite3(d);
    float e = -1.0f;
    if (q.use_cull || node32) {
        const CullRay cr = make_cull_ray(S, member, o, d);
        ww.cr_a[lane] = make_float4(cr.ox, cr.oy, cr.oz, cr.delta);
        ww.cr_b[lane] = make_float4(cr.ix, cr.iy, cr.iz, 0.0f);
        NodeRay nr;
        if (node32 && make_node_ray(S, cr, nr)) e = nr.e;
    }
    ww.e[lane] = e;
    ww.od[0][lane] = o.x; ww.od[1][lane] = o.y; ww.od[2][lane] = o.z;
    ww.od[3][lane] = d.x; ww.od[4][lane] = d.y; ww.od[5][lane] = d.z;
    q.best_t = CUDART_INF;
    q.best_obj = -1;
    q.best_e = -1;
    q.err = 0;
    q.ref = kNone;
    q.sp = q.untested = 1;
    q.slot = q.slot_end = 0;
    stack[0] = S.m_ref[member < 0 ? 0 : member];
}

// The lane's ray of the FP32 node test for its query so far, from its slot:
// formed anew for each stretch of the walk, so that no register holds it
// through the stage 1s (e < 0: nodes are tested in FP64).
__device__ __forceinline__ NodeRay work_node_ray(const WarpWork& w, int lane, double best_t) {
    const CullRay c = work_cull_ray(w, lane);
    NodeRay r;
    r.ix = c.ix; r.iy = c.iy; r.iz = c.iz;
    r.px = -c.ox * c.ix; r.py = -c.oy * c.iy; r.pz = -c.oz * c.iz;
    r.e = w.e[lane];
    r.e2 = 2.0f * r.e;
    r.set_best(best_t);
    return r;
}

// The FP64 node test of a lane's ray.
__device__ __forceinline__ bool work_box_exact(const WarpWork& w, int lane, const double* box, double best_t) {
    const V3 d = work_d(w, lane);
    const double inv[3] = { 1.0 / d.x, 1.0 / d.y, 1.0 / d.z };
    return ray_box_exact(work_o(w, lane), inv, box, best_t);
}

// Keeps the traversal state of a query that suspends for a Newton solve (the
// lane stands at the leaf slot of the patch being solved).
__device__ __forceinline__ void save_query(const WaveArgs& W, long long i, const AdvState& q, const int* stack) {
    int* qi = W.qs_int + i * kQsInt;
    if (!W.resume_queries || q.sp > kSaveStack) {
        qi[0] = -1;
        return;
    }
    qi[0] = q.sp;
    qi[1] = q.slot;
    qi[2] = q.slot_end;
    qi[3] = q.best_obj;
    qi[4] = q.best_e;
    W.qs_t[i] = q.best_t;
    int* st = W.qs_stack + i * kSaveStack;
    for (int k = 0; k < q.sp; ++k) st[k] = stack[k];
}

// Resumes a suspended query where it stopped (false when none was saved; the
// query then starts at the root).  The visit sequence is the one a replay from
// the root would produce, whose already-solved patches come from the resolved
// list.
__device__ __forceinline__ bool resume_query(const WaveArgs& W, long long i, AdvState& q, int* stack) {
    if (!W.resume_queries) return false;
    const int* qi = W.qs_int + i * kQsInt;
    const int sp = qi[0];
    if (sp < 0) return false;
    q.ref = kNone;
    q.sp = q.untested = sp;
    q.slot = qi[1];
    q.slot_end = qi[2];
    q.best_obj = qi[3];
    q.best_e = qi[4];
    q.best_t = W.qs_t[i];
    const int* st = W.qs_stack + i * kSaveStack;
    for (int k = 0; k < sp; ++k) stack[k] = st[k];
    return true;
}

// Triangle tests of the cells in w.cell: six per cell, 32 at a time over the
// whole batch.  A hit goes to the lane that owns the patch, which keeps the
// (t, key) minimum.
template <bool STATS>
__device__ __forceinline__ void batch_tris(const DScene& S, WarpWork& w, int n_cells, int lane, Stage1& mine) {
    const int n = S.coarse_n, nc = n - 1;
    const int total = 6 * n_cells;
    for (int p0 = 0; p0 < total; p0 += 32) {
        const int p = p0 + lane;
        Stage1 s;
        int owner = 0;
        if (p < total) {
            const int ce = p / 6, e = w.cell[ce];
            owner = e >> 8;
            const int pidx = __float_as_int(w.cr_b[owner].w);
            stage1_tri(S.c_xyz + static_cast<long long>(pidx) * n * n * 3,
                       S.c_cell + static_cast<long long>(pidx) * nc * nc * 4, n, (e >> 4) & 15, e & 15, p - 6 * ce,
                       work_o(w, owner), work_d(w, owner), s);
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

// Stage 1 of every lane of `batch` (patches of at most 4 x 4 blocks of 4 x 4
// cells), as three work lists over the whole warp: the block boxes of two
// patches at a time (16 lanes each), the cell boxes of two passing blocks at a
// time, the triangles of all passing cells 32 at a time.  Each list is
// compacted by ballot, so no lane idles because its own patch has little left.
template <bool STATS>
__device__ __forceinline__ void batch_stage1(const DScene& S, WarpWork& w, unsigned batch, int lane, Stage1& mine) {
    const int nc = S.coarse_n - 1, NB = S.n_blocks_side, NB2 = NB * NB;
    const unsigned lt = (1u << lane) - 1u;
    const int half = lane >> 4, hl = lane & 15;
    const int P = __popc(batch);
    mine.have = false;
    if (batch >> lane & 1u) w.lane_of[__popc(batch & lt)] = static_cast<unsigned char>(lane);
    if (STATS) w.cells[lane] = w.tris[lane] = 0;
    __syncwarp();
    const int hi = hl / NB, hj = hl - hi * NB;
    int n_blk = 0;
    for (int p = 0; p < P; p += 2) {
        const int c = p + half;
        const int owner = c < P && hl < NB2 ? w.lane_of[c] : -1;
        bool pass = false;
        if (owner >= 0) {
            const int pidx = __float_as_int(w.cr_b[owner].w);
            pass = cull_box(S.c_block_box + (static_cast<long long>(pidx) * NB2 + hl) * 6, work_cull_ray(w, owner));
        }
        const unsigned m = __ballot_sync(kFull, pass);
        if (pass) w.blk[n_blk + __popc(m & lt)] = static_cast<unsigned short>(owner << 8 | hi << 4 | hj);
        n_blk += __popc(m);
    }
    __syncwarp();
    int n_cell = 0;
    for (int p = 0; p < n_blk; p += 2) {
        const int c = p + half;
        int entry = 0;   // owner << 8 | row << 4 | column
        bool pass = false;
        if (c < n_blk) {
            const int e = w.blk[c], owner = e >> 8, i = ((e >> 4) & 15) * 4 + (hl >> 2), j = (e & 15) * 4 + (hl & 3);
            if (i < nc && j < nc) {
                entry = (e & ~255) | i << 4 | j;
                if (STATS) atomicAdd(&w.cells[owner], 1);
                const int pidx = __float_as_int(w.cr_b[owner].w);
                pass = cull_box(S.c_cell_box + (static_cast<long long>(pidx) * nc * nc + i * nc + j) * 6, work_cull_ray(w, owner));
                if (STATS && pass) atomicAdd(&w.tris[owner], 6);
            }
        }
        const unsigned m = __ballot_sync(kFull, pass);
        if (pass) w.cell[n_cell + __popc(m & lt)] = static_cast<unsigned short>(entry);
        n_cell += __popc(m);
        if (n_cell > kCellFlush && p + 2 < n_blk) {
            __syncwarp();
            batch_tris<STATS>(S, w, n_cell, lane, mine);
            __syncwarp();
            n_cell = 0;
        }
    }
    __syncwarp();
    batch_tris<STATS>(S, w, n_cell, lane, mine);
}

// Persistent: a lane owns a ray, walks its query to the next patch whose box
// the ray meets, and the warp runs the stage 1s of all its waiting lanes as one
// batch; a lane whose ray suspends or finishes fetches the next runnable ray.
// What bounds it: dependent loads of the walk (latency) and instruction issue
// of the batches, so the state kept in registers is small (origin, direction
// and cull ray of a lane live in shared memory for the batches) and the walk
// goes on until half of the lanes wait, which keeps the batches full.
//
// NT threads per block, MINB blocks per SM requested from the register
// allocator (launch shapes of the same body).
template <int NT, int MINB, bool STATS>
__global__ void __launch_bounds__(NT, MINB) k_advance(DScene S, TraceArgs A, WaveArgs W) {
    CountersT<STATS> ctr, cray;
    RayTallyT<STATS> tally;
    int i = -1, nres = 0, bounces = 0;
    int mode = M_IDLE;
    AdvState q;
    int stack[64];
    const int lane = threadIdx.x & 31;
    // Shared memory: the first S.smem_pairs node records (breadth-first order:
    // the top levels) and one WarpWork per warp.
    extern __shared__ __align__(16) float4 spair[];
    WarpWork& ww = reinterpret_cast<WarpWork*>(spair + 4 * S.smem_pairs)[threadIdx.x >> 5];
    for (int k = threadIdx.x; k < 4 * S.smem_pairs; k += blockDim.x) spair[k] = S.pair_rec[k];
    __syncthreads();
    const bool flat_ok = S.block_cells == 4 && S.n_blocks_side <= 4;
    // Runnable rays of this round: the host's count, or (graph-launched
    // trace) the count the previous round's control kernel left on the device.
    const long long n_run = W.count_dev ? static_cast<long long>(*W.count_dev) : W.n_runnable;
    // Rays per warp: in a round with fewer rays than the grid has lanes (the
    // late, small rounds) only the first ray_lanes lanes of each warp take rays
    // (the fewest, a power of two, that still cover the round), so the round is
    // spread over all the grid's warps instead of packed into a few full ones;
    // the other lanes only help with the stage 1s.
    int ray_lanes = 32;
    if (W.adapt_lanes) {
        const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
        const long long per = (n_run + warps - 1) / warps;
        while (ray_lanes > 1 && ray_lanes / 2 >= per) ray_lanes >>= 1;
    }
    if (lane >= ray_lanes) mode = M_DRAINED;
    // Watchdog: a launch that runs far past any real trace (W.watchdog_cycles
    // of SM clock, about 17 s by default) records an error and ends instead
    // of holding the GPU; checked on the first iteration and every 256th
    // after it.  Both exits of the loop are warp-uniform (this vote and the
    // drained vote at the end of the body); the inner loops end after at most
    // the nodes and slots of one query per lane.
    const long long t_start = clock64();
    unsigned int iter = 0;
    while (true) {
        if ((++iter & 255u) == 1u && __any_sync(kFull, clock64() - t_start > W.watchdog_cycles)) {
            if (lane == 0) atomicOr(&W.counters[3], 1u);
            break;
        }
        // ---- walk, and look through the leaves met, until half of the lanes with
        // a ray wait for something else
        const int half_alive = __popc(__ballot_sync(kFull, mode < M_IDLE)) >> 1;
        NodeRay nr = work_node_ray(ww, lane, q.best_t);
        do {
        while (__popc(__ballot_sync(kFull, mode == M_TRAV)) > half_alive) {
            if (mode == M_TRAV) {
                int ref = q.ref;
                if (ref == kNone && q.sp > 0) {
                    ref = stack[--q.sp];
                    if (q.sp < q.untested) {
                        // pushed before best_t was what it is: its own box again
                        q.untested = q.sp;
                        ++cray.node_tests;
                        const float* b32 = ref >= 0 ? S.node_box32 + 6LL * S.pair_node[ref]
                                                    : reinterpret_cast<const float*>(S.leaf_node + 2LL * ~ref);
                        int dec = nr.e >= 0.0f ? node_box_f32(b32, nr) : -1;
                        if (dec < 0) {
                            if (nr.e >= 0.0f) ++ctr.node_f64;
                            dec = work_box_exact(ww, lane, ref >= 0 ? S.node_box + 6LL * S.pair_node[ref] : S.leaf_box + 6LL * ~ref,
                                                 q.best_t);
                        }
                        if (!dec) ref = kNone;
                    }
                } else if (ref == kNone) {
                    mode = M_RESOLVE;
                }
                q.ref = kNone;
                if (ref >= 0) {
                    // both children (their records side by side); a child that fails now
                    // would fail when the reference pops it, best_t being no larger then
                    const float4* rec = ref < S.smem_pairs ? spair + 4 * ref : S.pair_rec + 4LL * ref;
                    const float4 a = rec[0], b = rec[1], c = rec[2], v = rec[3];
                    int l = -1, r = -1;
                    cray.node_tests += 2;
                    if (nr.e >= 0.0f) {
                        l = node_box_f32(a.x, a.y, a.z, a.w, b.x, b.y, nr);
                        r = node_box_f32(b.z, b.w, c.x, c.y, c.z, c.w, nr);
                        if (l < 0) ++ctr.node_f64;
                        if (r < 0) ++ctr.node_f64;
                    }
                    if ((l | r) < 0) {
                        const double* box = S.node_box + 6LL * __float_as_int(v.x);
                        if (l < 0) l = work_box_exact(ww, lane, box, q.best_t);
                        if (r < 0) r = work_box_exact(ww, lane, box + 6, q.best_t);
                    }
                    const bool right_first = (q.neg >> __float_as_int(v.w)) & 1u;
                    const int lref = __float_as_int(v.y), rref = __float_as_int(v.z);
                    if (l && r) {
                        q.ref = right_first ? rref : lref;
                        stack[q.sp++] = right_first ? lref : rref;   // depth of a median-split tree: at most 25
                    } else if (l || r) {
                        q.ref = l ? lref : rref;
                    }
                } else if (ref != kNone) {
                    const float4 b = S.leaf_node[2LL * ~ref + 1];
                    q.slot = __float_as_int(b.z);
                    q.slot_end = q.slot + __float_as_int(b.w);
                    mode = M_LEAF;
                }
            }
        }
        // ---- leaf slots of every lane at a leaf, each to its next patch whose
        // box the ray meets
        while (__ballot_sync(kFull, mode == M_LEAF)) {
            if (mode == M_LEAF) {
                if (q.slot >= q.slot_end) {
                    mode = M_TRAV;
                } else {
                    const LeafRec rec = load_leaf(S, q.slot);
                    if (rec.sub() < 0) {
                        QHit h;
                        if (triangle_intersect(S, ~rec.sub(), work_o(ww, lane), work_d(ww, lane), h, cray) && h.t < q.best_t) {
                            q.best_t = h.t;
                            nr.set_best(q.best_t);
                            q.untested = q.sp;
                            q.best_obj = rec.obj();
                            q.best_e = -1;
                        }
                        ++q.slot;
                    } else if (q.use_cull && !A.samples && !cull_leaf(rec, work_cull_ray(ww, lane))) {
                        // (while samples are recorded, a missed patch is a training sample)
                        ++cray.patch_tests;
                        ++cray.cell_tests;
                        ++q.slot;
                    } else {
                        const int obj = rec.obj();
                        int e = -1;
                        for (int k = 0; k < nres; ++k)
                            if (W.res_obj[static_cast<long long>(i) * kResolved + k] == obj) { e = k; break; }
                        if (e < 0) {
                            q.obj = obj;
                            ww.cr_b[lane].w = rec.b.z;
                            mode = M_S1;
                        } else {
                            const long long ei = static_cast<long long>(i) * kResolved + e;
                            q.err = W.res_err[ei];
                            if (q.err) {
                                q.best_e = e;
                                q.best_obj = obj;
                                mode = M_RESOLVE;
                            } else {
                                const double t = W.res_data[ei * kResData];
                                if (t < q.best_t) {
                                    q.best_t = t;
                                    nr.set_best(t);
                                    q.untested = q.sp;
                                    q.best_obj = obj;
                                    q.best_e = e;
                                }
                                ++q.slot;
                            }
                        }
                    }
                }
            }
        }
        } while (__popc(__ballot_sync(kFull, mode == M_TRAV)) > half_alive);
        // ---- stage 1 of every waiting lane
        const unsigned pend = __ballot_sync(kFull, mode == M_S1);
        if (pend) {
            const unsigned flat = flat_ok ? __ballot_sync(kFull, mode == M_S1 && q.use_cull) : 0u;
            if (flat) {
                __syncwarp();
                Stage1 res;
                batch_stage1<STATS>(S, ww, flat, lane, res);
                if (flat >> lane & 1u) {
                    q.s1 = res;
                    mode = M_S1_DONE;
                    ++cray.patch_tests;
                    if constexpr (STATS) {
                        cray.cell_tests += 1 + S.n_blocks_side * S.n_blocks_side + ww.cells[lane];
                        cray.tri_tests += ww.tris[lane];
                    }
                }
                __syncwarp();
            }
            // patches with more blocks or cells, and rays without culling: one
            // patch at a time by the whole warp
            for (unsigned rest = pend & ~flat; rest; rest &= rest - 1) {
                const int src = __ffs(rest) - 1;
                const bool scull = __shfl_sync(kFull, q.use_cull ? 1 : 0, src) != 0;
                CountersT<STATS> c2;
                const Stage1 res = warp_patch_stage1(S, __float_as_int(ww.cr_b[src].w), work_o(ww, src), work_d(ww, src),
                                                     scull, work_cull_ray(ww, src), lane, c2);
                long long pt = 0, ct = 0, tt = 0;
                if constexpr (STATS) {
                    pt = __shfl_sync(kFull, c2.patch_tests, 0);
                    ct = __shfl_sync(kFull, c2.cell_tests, 0);
                    tt = __shfl_sync(kFull, c2.tri_tests, 0);
                }
                if (lane == src) {
                    q.s1 = res;
                    cray.patch_tests += pt;
                    cray.cell_tests += ct;
                    cray.tri_tests += tt;
                    mode = M_S1_DONE;
                }
            }
        }
        NewtonRequest rq;
        if (mode == M_S1_DONE) {
            if (!q.s1.have) {
                if (A.samples)
                    record_sample(A, 0, work_o(ww, lane), work_d(ww, lane), __float_as_int(ww.cr_b[lane].w), 0.0, 0.0, 0.0);
                ++q.slot;
                mode = M_LEAF;
            } else if (nres >= kResolved) {
                mode = M_OVERFLOW;
            } else {
                W.res_obj[static_cast<long long>(i) * kResolved + nres] = q.obj;
                rq.ray = i;
                rq.entry = nres;
                rq.obj = q.obj;
                rq.key = q.s1.key;
                rq.t0 = q.s1.t;
                mode = M_SUSPEND;
            }
        } else if (mode == M_RESOLVE) {
            ++tally.queries;
            QHit h;
            h.err = q.err;
            h.obj = q.best_obj;
            h.ev0 = h.ev1 = 0.0;
            RayCtx r;
            r.o = work_o(ww, lane);
            r.d = work_d(ww, lane);
            r.member = A.ray_member ? A.ray_member[i] : -1;
            r.bounces = bounces;
            r.status = -1;
            r.err_obj = -1;
            r.ev0 = r.ev1 = 0.0;
            if (q.best_obj >= 0) {
                if (q.best_e >= 0) {
                    const double* rd = W.res_data + (static_cast<long long>(i) * kResolved + q.best_e) * kResData;
                    h.t = rd[0];
                    h.p = v3(rd[1], rd[2], rd[3]);
                    h.n = v3(rd[4], rd[5], rd[6]);
                    h.u = rd[7];
                    h.v = rd[8];
                    h.ev0 = rd[9];
                    h.ev1 = rd[10];
                } else {
                    CountersT<false> dummy;
                    triangle_intersect(S, S.obj_sub[q.best_obj], r.o, r.d, h, dummy);
                }
            }
            nres = 0;
            const bool on = step_ray(S, A, i, r, h);
            bounces = r.bounces;
            if (on && bounces < A.max_bounces) {
                adv_start_query(S, A, W, r.member, r.o, r.d, lane, ww, q, stack);
                mode = M_TRAV;
            } else {
                if (on) r.status = BBRT_RAY_MAX_BOUNCES;
                finish_ray(A, i, r);
                tally.bounces += bounces;
                tally.hist[r.status]++;
                mode = M_FINISH;
            }
        }
        // Only when some lane's ray left its working modes (one vote in the
        // common case): retire suspended / overflowed / finished rays, then
        // let idle lanes fetch the next runnable ray.
        if (__ballot_sync(kFull, mode >= M_FINISH && mode != M_DRAINED) != 0u) {
            // requests, overflows and the rays the free lanes take: three
            // counters, one round trip
            const unsigned m_req = __ballot_sync(kFull, mode == M_SUSPEND), m_ovf = __ballot_sync(kFull, mode == M_OVERFLOW);
            const unsigned m_new = __ballot_sync(kFull, mode >= M_FINISH && mode != M_DRAINED);
            unsigned at = 0;
            if (lane < 3) {
                const int add = __popc(lane == 0 ? m_req : lane == 1 ? m_ovf : m_new);
                if (add) at = atomicAdd(&W.counters[lane], static_cast<unsigned>(add));
            }
            const unsigned before = (1u << lane) - 1u;
            const unsigned rs = __shfl_sync(kFull, at, 0) + __popc(m_req & before);
            const unsigned os = __shfl_sync(kFull, at, 1) + __popc(m_ovf & before);
            const unsigned fs = __shfl_sync(kFull, at, 2) + __popc(m_new & before);
            if (mode == M_SUSPEND) W.req[rs] = rq;
            if (mode == M_OVERFLOW) W.overflow[os] = i;
            if (mode == M_SUSPEND || mode == M_OVERFLOW || mode == M_FINISH) {
                add_ray_work(A, i, cray);
                ctr.node_tests += cray.node_tests;
                ctr.patch_tests += cray.patch_tests;
                ctr.cell_tests += cray.cell_tests;
                ctr.tri_tests += cray.tri_tests;
                if (mode != M_FINISH) {
                    RayCtx r;
                    r.o = work_o(ww, lane);
                    r.d = work_d(ww, lane);
                    r.bounces = bounces;
                    save_ray(W, i, r, mode == M_SUSPEND ? nres + 1 : nres);
                    if (mode == M_SUSPEND) save_query(W, i, q, stack);
                }
                mode = M_IDLE;
            }
            if (mode == M_IDLE) {
                if (fs < n_run) {
                    cray = CountersT<STATS>();
                    nres = 0;
                    RayCtx r;
                    if (W.runnable == nullptr) {
                        i = W.order ? W.order[fs] : static_cast<int>(fs);
                        init_outputs(A, i);
                        r = start_ray(A, i);
                    } else {
                        i = W.runnable[fs].ray;
                        r = load_ray(A, W, i, nres);
                    }
                    bounces = r.bounces;
                    mode = M_TRAV;
                    if (r.status < 0) {
                        adv_start_query(S, A, W, r.member, r.o, r.d, lane, ww, q, stack);
                        if (W.runnable != nullptr && resume_query(W, i, q, stack)) mode = M_LEAF;
                        else if (r.bounces >= A.max_bounces) r.status = BBRT_RAY_MAX_BOUNCES;
                    }
                    if (r.status >= 0) {
                        finish_ray(A, i, r);
                        tally.bounces += r.bounces;
                        tally.hist[r.status]++;
                        mode = M_FINISH;
                    }
                } else {
                    mode = M_DRAINED;
                }
            }
            __syncwarp();
        }
        if (__all_sync(kFull, mode == M_DRAINED)) break;
    }
    flush_stats(A, ctr, tally);
}

template <int NT, int MINB, bool STATS>
cudaError_t launch_advance_stats(const DScene& Sl, const TraceArgs& A, const WaveArgs& W, int sm_count,
                                 cudaStream_t stream) {
    const size_t smem = static_cast<size_t>(Sl.smem_pairs) * 64 + (NT / 32) * sizeof(WarpWork);
    cudaError_t e = cudaFuncSetAttribute(k_advance<NT, MINB, STATS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_advance<NT, MINB, STATS>, NT, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    // A small round (the late ones) is spread over every SM: with full blocks
    // whose warps take fewer rays each (W.adapt_lanes, see k_advance), else
    // with smaller blocks rather than packed into the first few SMs.
    int threads = NT;
    long long blocks = static_cast<long long>(per_sm) * sm_count;
    if (W.adapt_lanes) {
        const long long need = (W.n_runnable + NT / 32 - 1) / (NT / 32);   // one ray per warp at least
        if (blocks > need) blocks = need;
    } else {
        const long long per_block = (W.n_runnable + static_cast<long long>(per_sm) * sm_count - 1) /
                                    (static_cast<long long>(per_sm) * sm_count);
        if (per_block < NT) threads = static_cast<int>(std::max<long long>(32, (per_block + 31) / 32 * 32));
        const long long need = (W.n_runnable + threads - 1) / threads;
        if (blocks > need) blocks = need;
    }
    k_advance<NT, MINB, STATS><<<static_cast<unsigned>(blocks), threads, smem, stream>>>(Sl, A, W);
    return cudaGetLastError();
}

// `budget`: dynamic shared memory a block may use; what the warps' work areas
// leave of it holds node records.  The statistics-free instance unless the call collects statistics or
// a per-ray work profile.
template <int NT, int MINB>
cudaError_t launch_advance_shape(const DScene& S, const TraceArgs& A, const WaveArgs& W, int sm_count, int budget,
                                 cudaStream_t stream) {
    DScene Sl = S;
    const int room = (budget - (NT / 32) * static_cast<int>(sizeof(WarpWork))) / 64;
    Sl.smem_pairs = std::min(S.n_pairs, std::max(room, 0));
    if (A.stats || A.ray_work) return launch_advance_stats<NT, MINB, true>(Sl, A, W, sm_count, stream);
    return launch_advance_stats<NT, MINB, false>(Sl, A, W, sm_count, stream);
}

}  // namespace

// Launch shapes of k_advance: 0 = 128 threads x 3 blocks per SM,
// 1 = 256 threads x 2 blocks per SM, 2 = 128 threads x 4 blocks per SM,
// 3 / 4 / 5 / 6 = 512 / 768 / 1024 / 384 threads x 1 block per SM.
cudaError_t launch_advance(const DScene& S, const TraceArgs& A, const WaveArgs& W, int sm_count, int shape,
                           cudaStream_t stream) {
    if (W.n_runnable <= 0) return cudaSuccess;
    constexpr int kSm = 227 * 1024;   // shared memory of an SM available to blocks (1 KB of it per block reserved)
    switch (shape) {
        case 1: return launch_advance_shape<256, 2>(S, A, W, sm_count, kSm / 2 - 1024, stream);
        case 2: return launch_advance_shape<128, 4>(S, A, W, sm_count, kSm / 4 - 1024, stream);
        case 3: return launch_advance_shape<512, 1>(S, A, W, sm_count, kSm, stream);
        case 4: return launch_advance_shape<768, 1>(S, A, W, sm_count, kSm, stream);
        case 5: return launch_advance_shape<1024, 1>(S, A, W, sm_count, kSm, stream);
        case 6: return launch_advance_shape<384, 1>(S, A, W, sm_count, kSm, stream);
        default: return launch_advance_shape<128, 3>(S, A, W, sm_count, kSm / 3 - 1024, stream);
    }
}

}  // namespace bbrt
