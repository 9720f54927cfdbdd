// Warp-per-ray trace and query kernels: 32 lanes work on one ray.
//
// Used where a ray's latency counts more than the number of rays in flight:
// small and middle batches, single queries, the last rays of a wavefront
// trace and rays whose query overflowed its resolved list.  Compiled with
// -fmad=false like the rest of the trace path (see exact.cuh).
//
// A query does not walk the tree.  BVH::intersect visits the leaves whose box
// passes with the best t at the time they are popped, in depth-first order;
// an ancestor's box contains the leaf's, and IEEE subtraction and
// multiplication are monotonic, so an ancestor passes whenever the leaf does
// (a slab time that is NaN, 0 * inf, is ignored by the test, for the leaf and
// for an ancestor that shares the face alike), and best t only falls.  So the
// visited leaves are those whose own box passes, in the order of their
// depth-first rank for the signs of the ray's direction (leaf_rank).  The
// lanes find them side by side:
//   1. subtrees of at most 32 leaves (cut_rec), 32 boxes at a time;
//   2. the leaves of a passing subtree, one per lane, the FP32 test with the
//      FP64 one where it does not decide; sorted by rank;
//   3. the leaves' slots, one per lane: the patches whose box the ray meets;
//   4. stage 1 of all of those at once: block boxes, cell boxes and triangles
//      as compacted work lists;
//   5. the stage-1 hits in order, a leaf's box tested again with the best t found
//      before it, so that what the reference would not have visited (behind a
//      nearer hit) changes nothing; Newton by the whole warp.
// Stage 1 behind the first hit is wasted, but a query is a handful of dependent
// steps instead of one per node and box level.
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

constexpr int kWarps = 4;           // warps per block
// Blocks per SM asked of the register allocator: 3 leaves 168 registers, 4 (128,
// three times the spills) measured slower: 4,096 tetrahedron rays 171 against
// 154 us, 96 queries 64 against 55 us.
constexpr int kMinBlocks = 3;
constexpr int kLeafCap = 64;        // leaves one query may visit here (more: warp_bvh_query)
constexpr int kSlotCap = 256;       // ... and their slots
constexpr int kListCap = 96;        // blocks and cells waiting to be tested
constexpr int kAxis = 8;            // nodes per axis of warp_newton

// One warp's shared memory.
struct RayWork {
    int rank[kLeafCap], leaf[kLeafCap];   // passing leaves as found
    int order[kLeafCap];                  // leaves in visiting order
    int slot[kSlotCap];                   // their slots in order
    unsigned char slot_leaf[kSlotCap];    // position of a slot's leaf in order[]
    int sub[32], obj[32], leaf_pos[32];   // candidates: patch or ~triangle, object, position in order[]
    int blk[kListCap], cell[kListCap];    // candidate << 24 | block or cell
    // Newton: barycentric basis (u, then v from kAxis on), rows' sums, evaluated fields
    double basis[2 * kAxis], rows[kAxis * 9], eval[9];
};

// node_box_f32 on a record's box.
__device__ __forceinline__ int rec_box_f32(const float4& a, const float4& b, const NodeRay& r) {
    return node_box_f32(a.x, a.y, a.z, a.w, b.x, b.y, r);
}

// BVH::intersect by walking the tree with a whole warp (every lane returns the
// same result): rays that are not finite, scenes without the FP32 node test's
// bounds, and queries that pass more leaves than the lists hold.
// TRIS, here and below: the scene has triangles.  Their tests in the same kernel
// cost a scene of patches 2 to 3 % (30,000 tetrahedron rays 0.653 ms against 0.639,
// queries 0.338 against 0.328), by the code they add.
template <bool TRIS, class Ctr>
__device__ QHit warp_bvh_query(const DScene& S, const V3& o, const V3& d, int cull_flag, int lane, Ctr& ctr,
                               bool off_patch_miss, int member) {
    QHit best;
    best.obj = -1;
    best.err = 0;
    best.t = CUDART_INF;
    const double inv[3] = { 1.0 / d.x, 1.0 / d.y, 1.0 / d.z };
    const bool neg[3] = { inv[0] < 0.0, inv[1] < 0.0, inv[2] < 0.0 };
    const bool use_cull = cull_ok(S, member, cull_flag, o, d);
    CullRay cr;
    if (use_cull) cr = make_cull_ray(S, member, o, d);
    double best_t = CUDART_INF;
    int stack[64];
    int sp = 0;
    stack[sp++] = root_node(S, member);
    while (sp > 0) {
        const int idx = stack[--sp];
        if (lane == 0) ++ctr.node_tests;
        if (!ray_box_exact(o, inv, S.node_box + 6LL * idx, best_t)) continue;
        const int* link = S.node_link + 4LL * idx;
        if (link[1] < 0) {
            const int start = link[0], count = link[2];
            for (int k = 0; k < count; ++k) {
                const LeafRec rec = load_leaf(S, start + k);
                const int obj = rec.obj(), sub = rec.sub();
                QHit h;
                h.err = 0;
                h.ev0 = h.ev1 = 0.0;
                int r = 0;
                if (!TRIS || sub >= 0) {
                    const Stage1 s1 = warp_patch_stage1(S, sub, o, d, use_cull, cr, lane, ctr);
                    if (s1.have) {
                        double u0, v0;
                        key_to_uv(S, s1.key, u0, v0);
                        long long it = 0;
                        r = newton_exact_j<0>(S, sub, o, d, u0, v0, s1.t, h, it);
                        if (lane == 0) ctr.newton_iters += it;
                    }
                } else {
                    CountersT<false> dummy;
                    r = triangle_intersect(S, ~sub, o, d, h, dummy);
                }
                if (off_patch_miss && h.err == BBRT_RAY_NEWTON_DOMAIN) {
                    if (lane == 0) ++ctr.off_patch;
                    continue;
                }
                if (h.err) {
                    h.obj = obj;
                    return h;
                }
                if (r && h.t < best_t) {
                    best_t = h.t;
                    best = h;
                    best.obj = obj;
                }
            }
            continue;
        }
        if (sp + 2 > 64) {
            best.err = BBRT_RAY_STACK_OVERFLOW;
            best.obj = -1;
            return best;
        }
        const int left = link[0], right = link[1];
        if (neg[link[3]]) { stack[sp++] = left; stack[sp++] = right; }
        else              { stack[sp++] = right; stack[sp++] = left; }
    }
    return best;
}

// Fields first[0] .. first[0] + 2 and so on (NF of them, in threes) of a patch at
// the basis in w.basis, into w.eval: a lane forms a row's sum over j of one
// field, then a lane per field adds the rows in order, skipping rows whose
// basis is 0 (eval_fields' sums in eval_fields' order).
template <int NF>
__device__ __forceinline__ void warp_eval(const double* __restrict__ F, int I, int J, RayWork& w, int lane) {
    for (int p = lane; p < I * NF; p += 32) {
        const int i = p / NF, f = p - i * NF;
        const double* row = F + static_cast<long long>(i) * J * 12 + (NF == 6 && f >= 3 ? f + 6 : f);
        double s = 0.0;
        if (w.basis[i] != 0.0)
            for (int j = 0; j < J; ++j) s += w.basis[kAxis + j] * row[j * 12];
        w.rows[p] = s;
    }
    __syncwarp();
    if (lane < NF) {
        double e = 0.0;
        for (int i = 0; i < I; ++i) {
            const double li = w.basis[i];
            if (li != 0.0) e += li * w.rows[i * NF + lane];
        }
        w.eval[lane] = e;
    }
    __syncwarp();
}

// Both axes' barycentric bases (basis_1d) into w.basis: lanes 0-7 of each
// half-warp take the u nodes, lanes 8-15 the v nodes.
// `node`, `weight`: the lane's own (of N on its axis).
__device__ __forceinline__ void warp_basis(double node, double weight, int N, double x, RayWork& w, int lane) {
    const int k = lane & (kAxis - 1), base = lane & kAxis;
    const bool mine = k < N;
    const double gap = mine ? x - node : 1.0;
    const unsigned on = __ballot_sync(kFull, mine && fabs(gap) < 1.0e-12) >> base & 0xFFu;
    const double li = mine ? weight / gap : 0.0;
    double denom = 0.0;
#pragma unroll
    for (int i = 0; i < kAxis; ++i) {
        const double x_i = __shfl_sync(kFull, li, base + i);
        if (i < N) denom += x_i;
    }
    const double b = on ? (k == __ffs(on) - 1 ? 1.0 : 0.0) : (mine ? li / denom : 0.0);
    if (lane < 2 * kAxis) w.basis[lane] = b;
    __syncwarp();
}

// newton_exact by the whole warp, for patches of at most 8 nodes per axis: the
// same operations in the same order, so the same result, on every lane.  A
// query rarely has more than one solve that counts, so the lanes share one
// solve (63 row sums of 7 nodes for the nine fields) instead of an 8-lane group
// each: 8-lane groups spent 126 shuffles an iteration on adding the rows up.
__device__ __forceinline__ int warp_newton(const DScene& S, int pidx, const V3 o, const V3 d, double u, double v, double t,
                                           QHit& h, long long& iters, RayWork& w, int lane) {
    const int I = S.p_dims[2 * pidx], J = S.p_dims[2 * pidx + 1];
    const double* un = S.p_nodes + S.p_node_off[pidx];   // un[I] vn[J] uw[I] vw[J]
    const bool v_axis = (lane & kAxis) != 0;
    const int N = v_axis ? J : I, k = min(lane & (kAxis - 1), N - 1) + (v_axis ? I : 0);
    const double node = un[k], weight = un[I + J + k];
    const double* F = S.p_fields + S.p_field_off[pidx];
    double step = CUDART_INF;
    for (int it = 0; it < S.newton_max_iters; ++it) {
        ++iters;
        warp_basis(node, weight, N, v_axis ? v : u, w, lane);
        warp_eval<9>(F, I, J, w, lane);
        double e[9];
#pragma unroll
        for (int f = 0; f < 9; ++f) e[f] = w.eval[f];
        const V3 R = v3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
        const double Fx = e[0] - R.x, Fy = e[1] - R.y, Fz = e[2] - R.z;
        const double a11 = e[3], a12 = e[6], a13 = -d.x;
        const double a21 = e[4], a22 = e[7], a23 = -d.y;
        const double a31 = e[5], a32 = e[8], a33 = -d.z;
        const double det = a11 * (a22 * a33 - a23 * a32) - a12 * (a21 * a33 - a23 * a31) + a13 * (a21 * a32 - a22 * a31);
        if (fabs(det) < 1e-14) { h.err = BBRT_RAY_NEWTON_SINGULAR; return 0; }
        const double d0 = Fx * (a22 * a33 - a23 * a32) - a12 * (Fy * a33 - a23 * Fz) + a13 * (Fy * a32 - a22 * Fz);
        const double d1 = a11 * (Fy * a33 - a23 * Fz) - Fx * (a21 * a33 - a23 * a31) + a13 * (a21 * Fz - Fy * a31);
        const double d2 = a11 * (a22 * Fz - Fy * a32) - a12 * (a21 * Fz - Fy * a31) + Fx * (a21 * a32 - a22 * a31);
        const double x0 = d0 / det, x1 = d1 / det, x2 = d2 / det;
        u -= x0;
        v -= x1;
        t -= x2;
        step = sqrt(x0 * x0 + x1 * x1 + x2 * x2);
        if (step < S.newton_tol) break;
    }
    if (step >= S.newton_tol) { h.err = BBRT_RAY_NEWTON_NOCONV; h.ev0 = step; return 0; }
    if (u < -1.0 - 1e-6 || u > 1.0 + 1e-6 || v < -1.0 - 1e-6 || v > 1.0 + 1e-6) {
        h.err = BBRT_RAY_NEWTON_DOMAIN; h.ev0 = u; h.ev1 = v; return 0;
    }
    warp_basis(node, weight, N, v_axis ? v : u, w, lane);
    warp_eval<6>(F, I, J, w, lane);   // point and normal
    h.t = t;
    h.p = v3(w.eval[0], w.eval[1], w.eval[2]);
    h.n = vnormalize(v3(w.eval[3], w.eval[4], w.eval[5]));
    h.u = u;
    h.v = v;
    return 1;
}

// Stage 1 of the P candidates in w.sub (patches; triangles are left to the
// caller), all with the same ray: lane c returns candidate c's winner.
template <class Ctr>
__device__ __forceinline__ Stage1 ray_stage1(const DScene& S, RayWork& w, int P, const V3& o, const V3& d, bool use_cull,
                                             const CullRay& cr, int lane, Ctr& ctr) {
    const int n = S.coarse_n, nc = n - 1;
    const unsigned lt = (1u << lane) - 1u;
    Stage1 mine;
    if (!use_cull) {
        const int total = nc * nc * 6;
        for (int c = 0; c < P; ++c) {
            const int sub = w.sub[c];
            if (sub < 0) continue;
            const double* X = S.c_xyz + static_cast<long long>(sub) * n * n * 3;
            const double* CC = S.c_cell + static_cast<long long>(sub) * nc * nc * 4;
            Stage1 s;
            for (int p = lane; p < total; p += 32) stage1_tri(X, CC, n, (p / 6) / nc, (p / 6) % nc, p % 6, o, d, s);
            warp_min_stage1(s);
            if (lane == c) mine = s;
            if (lane == 0) ctr.tri_tests += total;
        }
        return mine;
    }
    const int B = S.block_cells, B2 = B * B, NB = S.n_blocks_side, NB2 = NB * NB;
    const int blocks = P * NB2;
    int n_blk = 0;
    for (int b0 = 0; b0 < blocks; b0 += 32) {
        const int x = b0 + lane, c = x / NB2, b = x - c * NB2;
        bool pass = x < blocks && w.sub[c] >= 0;
        if constexpr (Ctr::kOn) {
            const int k = __popc(__ballot_sync(kFull, pass));
            if (lane == 0) ctr.cell_tests += k;
        }
        if (pass) pass = cull_box(S.c_block_box + (static_cast<long long>(w.sub[c]) * NB2 + b) * 6, cr);
        const unsigned m = __ballot_sync(kFull, pass);
        if (pass) w.blk[n_blk + __popc(m & lt)] = c << 24 | b;
        n_blk += __popc(m);
        if (n_blk == 0 || (n_blk <= kListCap - 32 && b0 + 32 < blocks)) continue;
        __syncwarp();
        const int cells = n_blk * B2;
        int n_cell = 0;
        for (int c0 = 0; c0 < cells; c0 += 32) {
            const int y = c0 + lane, q = y / B2, k = y - q * B2;
            bool ok = y < cells;
            int cand = 0, cell = 0;
            if (ok) {
                const int e = w.blk[q], bb = e & 0xFFFFFF, bi = bb / NB, ki = k / B;
                const int i = bi * B + ki, j = (bb - bi * NB) * B + (k - ki * B);
                cand = e >> 24;
                cell = i * nc + j;
                ok = i < nc && j < nc;
            }
            if constexpr (Ctr::kOn) {
                const int t = __popc(__ballot_sync(kFull, ok));
                if (lane == 0) ctr.cell_tests += t;
            }
            if (ok) ok = cull_box(S.c_cell_box + (static_cast<long long>(w.sub[cand]) * nc * nc + cell) * 6, cr);
            const unsigned cm = __ballot_sync(kFull, ok);
            if (ok) w.cell[n_cell + __popc(cm & lt)] = cand << 24 | cell;
            n_cell += __popc(cm);
            if (n_cell == 0 || (n_cell <= kListCap - 32 && c0 + 32 < cells)) continue;
            __syncwarp();
            const int tris = 6 * n_cell;
            for (int p0 = 0; p0 < tris; p0 += 32) {
                const int p = p0 + lane;
                Stage1 s;
                int owner = 0;
                if (p < tris) {
                    const int ce = p / 6, e = w.cell[ce], cl = e & 0xFFFFFF, i = cl / nc;
                    owner = e >> 24;
                    const int sub = w.sub[owner];
                    stage1_tri(S.c_xyz + static_cast<long long>(sub) * n * n * 3,
                               S.c_cell + static_cast<long long>(sub) * nc * nc * 4, n, i, cl - i * nc, p - 6 * ce, o, d, s);
                }
                for (unsigned hits = __ballot_sync(kFull, s.have); hits; hits &= hits - 1) {
                    const int src = __ffs(hits) - 1;
                    const double t = __shfl_sync(kFull, s.t, src);
                    const int key = __shfl_sync(kFull, s.key, src);
                    const int to = __shfl_sync(kFull, owner, src);
                    if (lane == to) mine.consider(t, key);
                }
            }
            if (lane == 0) ctr.tri_tests += tris;
            n_cell = 0;
            __syncwarp();
        }
        n_blk = 0;
        __syncwarp();
    }
    return mine;
}

// The best hit of a query by the steps above; false (nothing decided) when the
// ray or the scene needs warp_bvh_query.  Every lane returns the same result.
template <bool TRIS, class Ctr>
__device__ __forceinline__ bool ray_query(const DScene& S, RayWork& w, const V3& o, const V3& d, int cull_flag, int lane,
                                          Ctr& ctr, bool off_patch_miss, int member, QHit& best) {
    if (!S.leaf_lists || !finite3(o) || !finite3(d)) return false;
    const unsigned lt = (1u << lane) - 1u;
    const double inv[3] = { 1.0 / d.x, 1.0 / d.y, 1.0 / d.z };
    const int oct = (inv[0] < 0.0 ? 1 : 0) | (inv[1] < 0.0 ? 2 : 0) | (inv[2] < 0.0 ? 4 : 0);
    const bool use_cull = cull_ok(S, member, cull_flag, o, d);
    const CullRay cr = make_cull_ray(S, member, o, d);
    NodeRay nr;
    const bool node32 = make_node_ray(S, cr, nr) && S.node_f32;
    // ---- leaves whose box the ray meets
    const int c_end = S.m_cut[member < 0 ? 1 : member + 1];
    int n_leaf = 0;
    for (int k0 = S.m_cut[member < 0 ? 0 : member]; k0 < c_end; k0 += 32) {
        const int k = k0 + lane;
        bool pass = false;
        int first = 0, count = 0;
        if (k < c_end) {
            const float4 a = S.cut_rec[2LL * k], b = S.cut_rec[2LL * k + 1];
            first = __float_as_int(b.z);
            count = __float_as_int(b.w);
            // only a filter: undecided subtrees are looked into
            pass = node32 ? rec_box_f32(a, b, nr) != 0 : ray_box_exact(o, inv, S.cut_box + 6LL * k, CUDART_INF);
        }
        if constexpr (Ctr::kOn) {
            if (lane == 0) ctr.node_tests += min(32, c_end - k0);
        }
        for (unsigned todo = __ballot_sync(kFull, pass); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const int l = __shfl_sync(kFull, first, src) + lane, cnt = __shfl_sync(kFull, count, src);
            bool in = false;
            int dec = 0;
            if (lane < cnt) {
                dec = node32 ? rec_box_f32(S.leaf_node[2LL * l], S.leaf_node[2LL * l + 1], nr) : -1;
                in = dec < 0 ? ray_box_exact(o, inv, S.leaf_box + 6LL * l, CUDART_INF) : dec != 0;
            }
            const unsigned m = __ballot_sync(kFull, in);
            if constexpr (Ctr::kOn) {
                const int f64 = __popc(__ballot_sync(kFull, node32 && dec < 0));
                if (lane == 0) {
                    ctr.node_tests += cnt;
                    ctr.node_f64 += f64;
                }
            }
            const int at = n_leaf + __popc(m & lt);
            if (in && at < kLeafCap) {
                w.rank[at] = S.leaf_rank[8LL * l + oct];
                w.leaf[at] = l;
            }
            n_leaf += __popc(m);
        }
    }
    best.obj = -1;
    best.err = 0;
    best.t = CUDART_INF;
    if (n_leaf == 0) return true;
    if (n_leaf > kLeafCap) return false;
    __syncwarp();
    // ---- in visiting order
    for (int e = lane; e < n_leaf; e += 32) {
        const int r = w.rank[e];
        int at = 0;
        for (int j = 0; j < n_leaf; ++j) at += w.rank[j] < r ? 1 : 0;
        w.order[at] = w.leaf[e];
    }
    __syncwarp();
    int n_slot = 0;
    for (int e0 = 0; e0 < n_leaf; e0 += 32) {
        const int e = e0 + lane;
        int first = 0, count = 0;
        if (e < n_leaf) {
            const float4 b = S.leaf_node[2LL * w.order[e] + 1];
            first = __float_as_int(b.z);
            count = __float_as_int(b.w);
        }
        int x = count;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFull, x, off);
            if (lane >= off) x += y;
        }
        for (int k = 0; k < count; ++k) {
            const int at = n_slot + x - count + k;
            if (at < kSlotCap) {
                w.slot[at] = first + k;
                w.slot_leaf[at] = static_cast<unsigned char>(e);
            }
        }
        n_slot += __shfl_sync(kFull, x, 31);
    }
    if (n_slot > kSlotCap) return false;
    __syncwarp();
    // ---- their objects, 32 at a time
    double best_t = CUDART_INF;
    int open = -1;   // leaf last admitted (position in order)
    for (int s0 = 0; s0 < n_slot; s0 += 32) {
        const int s = s0 + lane;
        bool cand = false;
        int pos = 0;
        LeafRec rec;
        if (s < n_slot) {
            pos = w.slot_leaf[s];
            rec = load_leaf(S, w.slot[s]);
            cand = (TRIS && rec.sub() < 0) || !use_cull || cull_leaf(rec, cr);
        }
        const unsigned m = __ballot_sync(kFull, cand);
        if constexpr (Ctr::kOn) {
            const int t = __popc(__ballot_sync(kFull, s < n_slot && rec.sub() >= 0));
            if (lane == 0) {
                ctr.patch_tests += t;
                if (use_cull) ctr.cell_tests += t;
            }
        }
        const int P = __popc(m);
        if (!P) continue;
        if (cand) {
            const int at = __popc(m & lt);
            w.sub[at] = rec.sub();
            w.obj[at] = rec.obj();
            w.leaf_pos[at] = pos;
        }
        __syncwarp();
        Stage1 mine = ray_stage1(S, w, P, o, d, use_cull, cr, lane, ctr);
        if (TRIS && lane < P && w.sub[lane] < 0) {   // triangles: a lane each
            double u, v;
            const double* tv = S.tri + static_cast<long long>(~w.sub[lane]) * 9;
            mine.have = mt_full(o, d, load3(tv), load3(tv + 3), load3(tv + 6), mine.t, u, v);
        }
        // ---- hits in order
        for (unsigned hits = __ballot_sync(kFull, lane < P && mine.have); hits; hits &= hits - 1) {
            const int c = __ffs(hits) - 1;
            const int lp = w.leaf_pos[c];
            if (lp != open) {
                if (best_t < CUDART_INF && !ray_box_exact(o, inv, S.leaf_box + 6LL * w.order[lp], best_t)) continue;
                open = lp;
            }
            const int sub = w.sub[c];
            const double t0 = __shfl_sync(kFull, mine.t, c);
            const int key = __shfl_sync(kFull, mine.key, c);
            if (TRIS && sub < 0 && !(t0 < best_t)) continue;
            QHit h;
            h.err = 0;
            h.ev0 = h.ev1 = 0.0;
            int r;
            if (!TRIS || sub >= 0) {
                double u0, v0;
                key_to_uv(S, key, u0, v0);
                long long it = 0;
                if (S.max_nodes <= kAxis) r = warp_newton(S, sub, o, d, u0, v0, t0, h, it, w, lane);
                else r = newton_exact_j<0>(S, sub, o, d, u0, v0, t0, h, it);
                if (lane == 0) ctr.newton_iters += it;
            } else {
                CountersT<false> dummy;
                r = triangle_intersect(S, ~sub, o, d, h, dummy);
            }
            if (off_patch_miss && h.err == BBRT_RAY_NEWTON_DOMAIN) {
                if (lane == 0) ++ctr.off_patch;
                continue;
            }
            if (h.err) {
                best = h;
                best.obj = w.obj[c];
                __syncwarp();
                return true;
            }
            if (r && h.t < best_t) {
                best_t = h.t;
                best = h;
                best.obj = w.obj[c];
            }
        }
        __syncwarp();
    }
    return true;
}

template <bool TRIS, class Ctr>
__device__ __forceinline__ QHit any_query(const DScene& S, RayWork& w, const V3& o, const V3& d, int cull_flag, int lane,
                                          Ctr& ctr, bool off_patch_miss, int member) {
    QHit h;
    h.ev0 = h.ev1 = 0.0;
    if (ray_query<TRIS>(S, w, o, d, cull_flag, lane, ctr, off_patch_miss, member, h)) return h;
    return warp_bvh_query<TRIS>(S, o, d, cull_flag, lane, ctr, off_patch_miss, member);
}

// Whole rays, one per warp at a time: all n rays of the call (fresh), or the
// saved rays of `reqs` / `rays`, whose current query starts again.  Rays are
// handed out one at a time, so a warp that drew a long chain takes no more.
template <bool STATS, bool TRIS>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_rays(DScene S, TraceArgs A, WaveArgs W, const NewtonRequest* reqs,
                                                         const int* rays, long long n) {
    __shared__ RayWork work[kWarps];
    RayWork& w = work[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const bool fresh = !reqs && !rays;
    if (W.count_dev) n = *W.count_dev;
    unsigned int* next = W.counters ? W.counters + (reqs ? kWcTailNext : kWcOvfNext) : nullptr;
    CountersT<STATS> ctr;
    RayTallyT<STATS> tally;
    while (true) {
        long long slot = 0;
        if (lane == 0) slot = next ? atomicAdd(next, 1u) : static_cast<long long>(atomicAdd(A.work_counter, 1ULL));
        slot = __shfl_sync(kFull, slot, 0);
        if (slot >= n) break;
        const long long i = fresh ? slot : reqs ? reqs[slot].ray : rays[slot];
        RayCtx r;
        if (fresh) {
            if (lane == 0) init_outputs(A, i);
            r = start_ray(A, i);
        } else {
            int nres;
            r = load_ray(A, W, i, nres);
        }
        CountersT<STATS> c1;
        if (A.query_out) {
            const QHit h = any_query<TRIS>(S, w, r.o, r.d, A.cull, lane, c1, false, r.member);
            if (lane == 0) write_hit(static_cast<bbrt_hit*>(A.query_out) + i, h);
            continue;
        }
        while (r.status < 0) {
            if (r.bounces >= A.max_bounces) { r.status = BBRT_RAY_MAX_BOUNCES; break; }
            if (lane == 0) ++tally.queries;
            const QHit h = any_query<TRIS>(S, w, r.o, r.d, A.cull, lane, c1, A.off_patch_miss != 0, r.member);
            if (!step_ray(S, A, i, r, h, lane == 0)) break;
        }
        if (lane == 0) {
            add_ray_work(A, i, c1);
            finish_ray(A, i, r);
            tally.bounces += r.bounces;
            tally.hist[r.status]++;
        }
        ctr.node_tests += c1.node_tests;
        ctr.patch_tests += c1.patch_tests;
        ctr.cell_tests += c1.cell_tests;
        ctr.tri_tests += c1.tri_tests;
        ctr.newton_iters += c1.newton_iters;
        ctr.off_patch += c1.off_patch;
        ctr.node_f64 += c1.node_f64;
    }
    flush_stats(A, ctr, tally, true);
}

// BVH queries, one per warp at a time.
template <bool TRIS>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_query_warp(DScene S, QueryArgs Q) {
    __shared__ RayWork work[kWarps];
    RayWork& w = work[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long long warps = static_cast<long long>(gridDim.x) * kWarps;
    for (long long i = static_cast<long long>(blockIdx.x) * kWarps + (threadIdx.x >> 5); i < Q.n; i += warps) {
        CountersT<false> ctr;
        const QHit r = any_query<TRIS>(S, w, load3(Q.origins + 3 * i), load3(Q.dirs + 3 * i), Q.cull, lane, ctr, false, -1);
        if (lane == 0) write_hit(static_cast<bbrt_hit*>(Q.out) + i, r);
    }
}

template <class K>
cudaError_t grid_for(K kernel, long long n, int sm_count, unsigned* blocks) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, 0);
    if (e != cudaSuccess) return e;
    *blocks = static_cast<unsigned>(std::min<long long>(static_cast<long long>(std::max(per_sm, 1)) * sm_count,
                                                        (n + kWarps - 1) / kWarps));
    return cudaSuccess;
}

}  // namespace

// Saved rays (`reqs` or `rays`), or with both null all n rays of the call.  The
// statistics-free instance unless the call collects statistics or a per-ray
// work profile.
cudaError_t launch_rays(const DScene& S, const TraceArgs& A, const WaveArgs& W, const NewtonRequest* reqs, const int* rays,
                        long long n, int sm_count, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    auto launch = [&](auto kernel) {
        unsigned blocks = 0;
        const cudaError_t e = grid_for(kernel, n, sm_count, &blocks);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, kWarps * 32, 0, stream>>>(S, A, W, reqs, rays, n);
        return cudaGetLastError();
    };
    if (A.stats || A.ray_work) return S.tri ? launch(k_rays<true, true>) : launch(k_rays<true, false>);
    return S.tri ? launch(k_rays<false, true>) : launch(k_rays<false, false>);
}

cudaError_t launch_query_warp(const DScene& S, const QueryArgs& Q, int sm_count, cudaStream_t stream) {
    if (Q.n <= 0) return cudaSuccess;
    auto launch = [&](auto kernel) {
        unsigned blocks = 0;
        const cudaError_t e = grid_for(kernel, Q.n, sm_count, &blocks);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, kWarps * 32, 0, stream>>>(S, Q);
        return cudaGetLastError();
    };
    return S.tri ? launch(k_query_warp<true>) : launch(k_query_warp<false>);
}

// Loads the kernels of launch_rays on the current device (see noalloc_prepare).
cudaError_t rays_prepare() {
    cudaFuncAttributes fa;
    for (auto kernel : { k_rays<true, true>, k_rays<true, false>, k_rays<false, true>, k_rays<false, false> }) {
        const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace bbrt
