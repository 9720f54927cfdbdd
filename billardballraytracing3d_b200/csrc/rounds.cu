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
        // a launch that runs far past any real round gives up (see advance.cu), the
        // whole warp at once: the lanes' clocks need not agree
        if (__any_sync(kFull, clock64() - t_start > W.watchdog_cycles)) {
            if (lane == 0) atomicOr(&W.counters[3], 1u);
            break;
        }
    }
    __syncwarp();
    flush_stats(A, ctr, tally);
}

// ---- stage 1 -----------------------------------------------------------------

constexpr int kRays = 16;           // rays of a warp
constexpr int kS1Warps = 4;         // warps per block
constexpr int kLeafLanes = 32;      // leaves expanded at a time
constexpr int kMaxCand = kLeafLanes * kSplitLeafSlots;
constexpr int kQueue = 80;          // nodes of a quadtree level that wait (at most 15 and 64 new ones)
constexpr int kBlkCap = 128, kCellCap = 64;   // larger grids: blocks and cells that wait

// A ray's cull test as fused multiply-adds: slab times fma(b, i, p) of the two
// faces of an axis, inflated, with p = -(o + delta) i for the min face and
// (delta - o) i for the max face.  Rounding: o, o + delta and the product in p
// 3 units of 2^-24 (|o| + delta) |i|, 1/d 2 of (|b| + |o| + delta) |i|, the sum
// 1: 6 (|b| + |o| + delta), as a distance, of the 32 that delta holds for the
// slab test (cull_constants).  |i| is kept to 1e18, which is sound on the axes
// that it cuts off (|d_a| < 1e-18): a triangle is hit only with |det| >= 1e-9, so
// |d| >= 1e-9 / h^2 (h: cull_h, at least the longest edge) and the hit's
// t <= 1e9 h^2 L; up to it the ray moves less than 1e-9 h^2 L on such an axis, and
// delta holds cull_a L = 2.8e-5 h^2 L, so the origin is that far inside the
// inflated slab and the times cut off still contain [0, t].
struct __align__(16) CullFma {
    float ix, iy, iz, nx, ny, nz, xx, xy, xz, pad[3];
};

// false: a value beyond the range the test is sound in (the ray then goes to the
// overflow list).
__device__ __forceinline__ bool make_cull_fma(const CullRay& c, CullFma& f) {
    f.ix = fminf(fmaxf(c.ix, -1e18f), 1e18f);
    f.iy = fminf(fmaxf(c.iy, -1e18f), 1e18f);
    f.iz = fminf(fmaxf(c.iz, -1e18f), 1e18f);
    f.nx = -(c.ox + c.delta) * f.ix; f.xx = (c.delta - c.ox) * f.ix;
    f.ny = -(c.oy + c.delta) * f.iy; f.xy = (c.delta - c.oy) * f.iy;
    f.nz = -(c.oz + c.delta) * f.iz; f.xz = (c.delta - c.oz) * f.iz;
    const float m = fmaxf(fmaxf(fmaxf(fabsf(f.nx), fabsf(f.xx)), fmaxf(fabsf(f.ny), fabsf(f.xy))),
                          fmaxf(fabsf(f.nz), fabsf(f.xz)));
    return m <= 1e37f;
}

__device__ __forceinline__ bool cull_fma(float x0, float y0, float z0, float x1, float y1, float z1, const CullFma& f) {
    float t1 = fmaf(x0, f.ix, f.nx), t2 = fmaf(x1, f.ix, f.xx);
    float tmin = fminf(t1, t2), tmax = fmaxf(t1, t2);
    t1 = fmaf(y0, f.iy, f.ny); t2 = fmaf(y1, f.iy, f.xy);
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    t1 = fmaf(z0, f.iz, f.nz); t2 = fmaf(z1, f.iz, f.xz);
    tmin = fmaxf(fmaxf(tmin, 0.0f), fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    return tmin <= tmax;
}

// One warp's shared memory.
struct __align__(16) S1Work {
    CullFma cull[kRays];                       // cull tests of the rays
    double od[6][kRays];                       // origins, directions
    int ray[kRays], n_hits[kRays], leaf0[kRays];
    unsigned char leaf_ray[kRays * kSplitLeaves];   // the leaves in (ray, visiting) order: their rays
    // candidates in that order: patch or ~triangle, slot, stage-1 winner (key < 0: none), ray, place of its leaf
    int sub[kMaxCand], slot[kMaxCand], key[kMaxCand];
    double t[kMaxCand];
    unsigned char cand_ray[kMaxCand], cand_pos[kMaxCand];
    int queue[4][kQueue];                      // quadtree nodes, then cells, that passed: candidate << 16 | Morton index
    int blk[kBlkCap];                          // larger grids: passing blocks, candidate << 24 | block ...
    int cell[kCellCap];                        // ... and cells
    int cells[kRays], tris[kRays];             // box and triangle tests (statistics)
};

// Cell (i, j) of Morton index m (j in the even bits).
__device__ __forceinline__ void morton_cell(int m, int& i, int& j) {
    j = (m & 1) | (m >> 1 & 2) | (m >> 2 & 4) | (m >> 3 & 8);
    m >>= 1;
    i = (m & 1) | (m >> 1 & 2) | (m >> 2 & 4) | (m >> 3 & 8);
}

// Triangle tests of up to sixteen cells: a lane takes one of a cell's two
// triangles at its three offsets (six lanes a cell loaded every corner three
// times and handed over three times the hits).  A candidate keeps its
// (t, key) minimum.
template <class Cell>
__device__ __forceinline__ void s1_tris(const DScene& S, S1Work& w, int n_cells, int lane, Cell cell_at) {
    const int n = S.coarse_n, nc = n - 1;
    Stage1 s;
    int cand = 0;
    if (lane < 2 * n_cells) {
        int i, j;
        cell_at(lane >> 1, cand, i, j);
        const int sub = w.sub[cand], r = w.cand_ray[cand];
        stage1_tri3(S.c_xyz + static_cast<long long>(sub) * n * n * 3, S.c_cell + static_cast<long long>(sub) * nc * nc * 4, n,
                    i, j, lane & 1, v3(w.od[0][r], w.od[1][r], w.od[2][r]), v3(w.od[3][r], w.od[4][r], w.od[5][r]), s);
    }
    for (unsigned hits = __ballot_sync(kFull, s.have); hits; hits &= hits - 1) {
        if (lane == __ffs(hits) - 1) {
            Stage1 b;
            b.key = w.key[cand];
            b.have = b.key >= 0;
            b.t = w.t[cand];
            b.consider(s.t, s.key);
            w.t[cand] = b.t;
            w.key[cand] = b.key;
        }
        __syncwarp();
    }
}

// Stage 1 of candidates [first, last) by their patches' quadtrees: every step
// takes sixteen waiting nodes of one level and tests their four children, two a
// lane, or sixteen cells' triangles; the deepest level with enough waiting goes
// first, so the lists stay short and the lanes full (5.3 tests a level and
// candidate where sixteen blocks and sixteen cells a block were 32).
template <bool STATS>
__device__ __forceinline__ void s1_quads(const DScene& S, S1Work& w, int first, int last, int lane) {
    const unsigned lt = (1u << lane) - 1u;
    int next = first, n1 = 0, n2 = 0, n3 = 0, n4 = 0;
    while (true) {
        int level;
        if (n4 >= 16) level = 4;
        else if (n3 >= 16) level = 3;
        else if (n2 >= 16) level = 2;
        else if (n1 >= 16) level = 1;
        else if (next < last) level = 0;
        else if (n1 > 0) level = 1;
        else if (n2 > 0) level = 2;
        else if (n3 > 0) level = 3;
        else if (n4 > 0) level = 4;
        else break;
        if (level == 4) {
            const int k = min(n4, 16), at = n4 - k;
            s1_tris(S, w, k, lane, [&](int e, int& cand, int& i, int& j) {
                const int x = w.queue[3][at + e];
                cand = x >> 16;
                morton_cell(x & 0xFFFF, i, j);
            });
            n4 = at;
            continue;
        }
        // two nodes' children per lane, their boxes in flight together
        const int have = level == 0 ? last - next : level == 1 ? n1 : level == 2 ? n2 : n3;
        const int k = min(have, 16);
        const int off = level == 0 ? 0 : level == 1 ? 4 : level == 2 ? 20 : 84;
        int entry[2], ray[2];
        float2 b[2][3];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int e = (lane >> 2) + 8 * u;
            ray[u] = -1;
            entry[u] = 0;
            if (e < k) {
                const int x = level == 0 ? (next + e) << 16 : w.queue[level - 1][have - k + e];
                const int cand = x >> 16, m = (x & 0xFFFF) * 4 + (lane & 3);
                entry[u] = cand << 16 | m;
                const int sub = w.sub[cand];
                if (sub >= 0) {
                    ray[u] = w.cand_ray[cand];
                    const float2* q = reinterpret_cast<const float2*>(S.quad_box) + (static_cast<long long>(sub) * kQuadNodes + off + m) * 3;
#pragma unroll
                    for (int a = 0; a < 3; ++a) b[u][a] = q[a];
                }
            }
        }
        int add = 0;
        int to = level == 0 ? n1 : level == 1 ? n2 : level == 2 ? n3 : n4;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            bool pass = ray[u] >= 0;
            if (pass) {
                if (STATS) atomicAdd(&w.cells[ray[u]], 1);
                pass = b[u][0].x <= b[u][1].y &&
                       cull_fma(b[u][0].x, b[u][0].y, b[u][1].x, b[u][1].y, b[u][2].x, b[u][2].y, w.cull[ray[u]]);
                if (STATS && pass && level == 3) atomicAdd(&w.tris[ray[u]], 6);
            }
            const unsigned pm = __ballot_sync(kFull, pass);
            if (pass) w.queue[level][to + add + __popc(pm & lt)] = entry[u];
            add += __popc(pm);
        }
        __syncwarp();
        if (level == 0) { next += k; n1 += add; }
        else if (level == 1) { n1 -= k; n2 += add; }
        else if (level == 2) { n2 -= k; n3 += add; }
        else { n3 -= k; n4 += add; }
    }
}

// The same for larger grids: a candidate's blocks, then the cells of the blocks
// that pass, flattened over the candidates.
template <bool STATS>
__device__ __forceinline__ void s1_blocks(const DScene& S, S1Work& w, int first, int last, int lane) {
    const int nc = S.coarse_n - 1, B = S.block_cells, B2 = B * B, NB = S.n_blocks_side, NB2 = NB * NB;
    const unsigned lt = (1u << lane) - 1u;
    int n_blk = 0, n_cell = 0;
    const long long blocks = static_cast<long long>(last - first) * NB2;
    auto flush = [&] {
        __syncwarp();
        for (int at = 0; at < n_cell; at += 16)
            s1_tris(S, w, min(16, n_cell - at), lane, [&](int e, int& cand, int& i, int& j) {
                const int x = w.cell[at + e];
                cand = x >> 24;
                i = (x & 0xFFFFFF) / nc;
                j = (x & 0xFFFFFF) - i * nc;
            });
        __syncwarp();
        n_cell = 0;
    };
    for (long long b0 = 0; b0 < blocks; b0 += 32) {
        const long long x = b0 + lane;
        const int c = first + static_cast<int>(x / NB2), b = static_cast<int>(x % NB2);
        bool pass = x < blocks;
        if (pass) {
            const int sub = w.sub[c], r = w.cand_ray[c];
            pass = sub >= 0;
            if (STATS && pass) atomicAdd(&w.cells[r], 1);
            if (pass) {
                const float2* q = reinterpret_cast<const float2*>(S.c_block_box + (static_cast<long long>(sub) * NB2 + b) * 6);
                pass = cull_fma(q[0].x, q[0].y, q[1].x, q[1].y, q[2].x, q[2].y, w.cull[r]);
            }
        }
        const unsigned m = __ballot_sync(kFull, pass);
        if (pass) w.blk[n_blk + __popc(m & lt)] = c << 24 | b;
        n_blk += __popc(m);
        if (b0 + 32 < blocks && n_blk <= kBlkCap - 32) continue;
        __syncwarp();
        const int cells = n_blk * B2;
        for (int y0 = 0; y0 < cells; y0 += 32) {
            const int y = y0 + lane, q = y / B2, k = y - q * B2;
            bool ok = y < cells;
            int cand = 0, cell = 0;
            if (ok) {
                const int e = w.blk[q], bb = e & 0xFFFFFF, bi = bb / NB, ki = k / B;
                const int i = bi * B + ki, j = (bb - bi * NB) * B + (k - ki * B);
                cand = e >> 24;
                cell = i * nc + j;
                ok = i < nc && j < nc;
            }
            if (ok) {
                const int r = w.cand_ray[cand];
                if (STATS) atomicAdd(&w.cells[r], 1);
                const float2* q2 = reinterpret_cast<const float2*>(S.c_cell_box +
                                                                   (static_cast<long long>(w.sub[cand]) * nc * nc + cell) * 6);
                ok = cull_fma(q2[0].x, q2[0].y, q2[1].x, q2[1].y, q2[2].x, q2[2].y, w.cull[r]);
                if (STATS && ok) atomicAdd(&w.tris[r], 6);
            }
            const unsigned cm = __ballot_sync(kFull, ok);
            if (ok) w.cell[n_cell + __popc(cm & lt)] = cand << 24 | cell;
            n_cell += __popc(cm);
            if (n_cell > kCellCap - 32) flush();
        }
        n_blk = 0;
        __syncwarp();
    }
    flush();
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
template <bool QUADS, bool STATS>
__global__ void __launch_bounds__(kS1Warps * 32, 4) k_stage1(DScene S, TraceArgs A, WaveArgs W, RoundControl R) {
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
        bool over = false;
        if (lane < rays) {
            i = W.listed[g + lane];
            count = W.n_leaves[i];
            const V3 o = load3(W.o + 3LL * i), d = load3(W.d + 3LL * i);
            CullFma f;
            over = !make_cull_fma(make_cull_ray(S, A.ray_member ? A.ray_member[i] : -1, o, d), f);
            w.cull[lane] = f;
            if (over) count = 0;
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
        // then stage 1 of them
        for (int l0 = 0; l0 < n_leaf; l0 += kLeafLanes) {
            int r = 0, first = 0, pos = 0;
            unsigned pass = 0;
            if (lane < kLeafLanes && l0 + lane < n_leaf) {
                r = w.leaf_ray[l0 + lane];
                pos = l0 + lane - w.leaf0[r];
                const int leaf = W.leaves[static_cast<long long>(w.ray[r]) * kSplitLeaves + pos];
                const float4 b = S.leaf_node[2LL * leaf + 1];
                first = __float_as_int(b.z);
                const int slots = __float_as_int(b.w);
                const CullFma f = w.cull[r];
                for (int k = 0; k < slots; ++k) {
                    const LeafRec rec = load_leaf(S, first + k);
                    if (rec.sub() < 0 || cull_fma(rec.a.x, rec.a.y, rec.a.z, rec.a.w, rec.b.x, rec.b.y, f)) pass |= 1u << k;
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
            int at = y - __popc(pass);
            for (unsigned m = pass; m; m &= m - 1, ++at) {
                const int slot = first + __ffs(m) - 1;
                w.sub[at] = __float_as_int(S.leaf_rec[2LL * slot + 1].z);
                w.slot[at] = slot;
                w.key[at] = -1;
                w.cand_ray[at] = static_cast<unsigned char>(r);
                w.cand_pos[at] = static_cast<unsigned char>(pos);
            }
            const int n_cand = __shfl_sync(kFull, y, 31);
            __syncwarp();
            if (QUADS) s1_quads<STATS>(S, w, 0, n_cand, lane);
            else s1_blocks<STATS>(S, w, 0, n_cand, lane);
            __syncwarp();
            // hits in visiting order
            for (int c0 = 0; c0 < n_cand; c0 += 32) {
                const int c = c0 + lane;
                bool hit = c < n_cand;
                double t = 0.0;
                int key = 0;
                if (hit) {
                    if (w.sub[c] < 0) {
                        const int q = w.cand_ray[c];
                        QHit h;
                        CountersT<false> dummy;
                        hit = triangle_intersect(S, ~w.sub[c], v3(w.od[0][q], w.od[1][q], w.od[2][q]),
                                                 v3(w.od[3][q], w.od[4][q], w.od[5][q]), h, dummy) != 0;
                        t = h.t;
                        ctr.tri_tests += 1;
                    } else {
                        key = w.key[c];
                        hit = key >= 0;
                        t = w.t[c];
                    }
                }
                const unsigned hm = __ballot_sync(kFull, hit);
                if (hit) {
                    const int q = w.cand_ray[c];
                    const unsigned peers = __match_any_sync(hm, q);
                    const int old = w.n_hits[q], place = old + __popc(peers & lt);
                    if (place < kSplitHits) {
                        SplitHit* out = W.hits + static_cast<long long>(w.ray[q]) * kSplitHits + place;
                        out->t = t;
                        out->obj = __float_as_int(S.leaf_rec[2LL * w.slot[c] + 1].w);
                        out->leaf = W.leaves[static_cast<long long>(w.ray[q]) * kSplitLeaves + w.cand_pos[c]];
                        out->key = key;
                    }
                    __syncwarp(hm);
                    if (lane == __ffs(peers) - 1) w.n_hits[q] = old + __popc(peers);
                }
                __syncwarp();
            }
        }
        // ---- each ray's first hit is its Newton request; none: it escapes
        bool ask = false;
        NewtonRequest rq;
        if (lane < rays && !over) {
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

template <bool QUADS, bool STATS>
cudaError_t launch_stage1(const DScene& S, const TraceArgs& A, const WaveArgs& W, const RoundControl& R, int sm_count,
                          cudaStream_t stream) {
    constexpr int smem = kS1Warps * sizeof(S1Work);
    cudaError_t e = cudaFuncSetAttribute(k_stage1<QUADS, STATS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int per_sm = 0;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage1<QUADS, STATS>, kS1Warps * 32, smem);
    if (e != cudaSuccess) return e;
    const long long blocks = std::min<long long>(static_cast<long long>(std::max(per_sm, 1)) * sm_count,
                                                 (W.n_runnable + kS1Warps - 1) / kS1Warps);
    k_stage1<QUADS, STATS><<<static_cast<unsigned>(blocks), kS1Warps * 32, smem, stream>>>(S, A, W, R);
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
    const bool stats = A.stats || A.ray_work, quads = S.quad_box != nullptr;
    const cudaError_t e = stats ? launch_walk<true>(S, A, W, sm_count, stream) : launch_walk<false>(S, A, W, sm_count, stream);
    if (e != cudaSuccess) return e;
    if (stats) return quads ? launch_stage1<true, true>(S, A, W, R, sm_count, stream) : launch_stage1<false, true>(S, A, W, R, sm_count, stream);
    return quads ? launch_stage1<true, false>(S, A, W, R, sm_count, stream) : launch_stage1<false, false>(S, A, W, R, sm_count, stream);
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
