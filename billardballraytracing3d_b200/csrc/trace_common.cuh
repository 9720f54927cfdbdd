// Device functions shared by the trace kernels (advance.cu, trace_kernels.cu):
// cull and node tests, SurfacePatch stage 1, per-thread queries and the
// bounce loop as per-ray state steps, all decisions in the reference's FP64
// arithmetic (see exact.cuh; both files are compiled with -fmad=false).
//
// Reference (manuelarturosantana/BillardBallRayTracing3D):
//   RayTracingDriver::trace_ray   include/RayTracingDriver.hpp:172-242
//   BVH::intersect                include/BVH.hpp:75-128
//   SurfacePatch::intersect       include/ScatObjects/SurfacePatch.hpp:253-303
//   Triangle::intersect           include/ScatObjects/Triangle.hpp:26-28
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>

#include "../../include/bbrt.h"
#include "exact.cuh"
#include "guess.h"

namespace bbrt {

// Work counters of the statistics, per thread (summed per warp at the end of
// a launch).  CountersT<false> holds nothing: a launch that collects no
// statistics (and no per-ray work profile) uses it, so the counting, its
// 64-bit registers and their spills compile away.
struct NoCount {
    __device__ __forceinline__ NoCount& operator++() { return *this; }
    __device__ __forceinline__ NoCount operator++(int) { return *this; }
    __device__ __forceinline__ NoCount& operator+=(long long) { return *this; }
    __device__ __forceinline__ operator long long() const { return 0; }
};

template <bool ON>
struct CountersT {
    static constexpr bool kOn = true;
    long long node_tests = 0, patch_tests = 0, cell_tests = 0, tri_tests = 0, newton_iters = 0;
    long long off_patch = 0;   // learned form: Newton roots outside their patch taken as misses
    long long node_f64 = 0;    // node tests the FP32 test left to the FP64 one
};
template <>
struct CountersT<false> {
    static constexpr bool kOn = false;
    NoCount node_tests, patch_tests, cell_tests, tri_tests, newton_iters, off_patch, node_f64;
};
using Counters = CountersT<true>;

// Per-ray data of the FP32 cull test (computed once per query).
struct CullRay {
    float ox, oy, oz, ix, iy, iz, delta;
};

__device__ __forceinline__ bool finite3(const V3& a) {
    return isfinite(a.x) && isfinite(a.y) && isfinite(a.z);
}

// Scene values of a ray's scene: the scene itself, or member m of a scene set.
__device__ __forceinline__ double scene_diag(const DScene& S, int m) {
    return m < 0 ? S.scene_diagonal : S.m_param[m * kMemberParams];
}
__device__ __forceinline__ int root_node(const DScene& S, int m) { return m < 0 ? 0 : S.m_root[m]; }

// The cull inflation bound is derived for |d| <= 1 (the trace loop always
// normalises d); single queries with longer or non-finite rays skip culling.
__device__ __forceinline__ bool cull_ok(const DScene& S, int m, int cull_flag, const V3& o, const V3& d) {
    const bool on = m < 0 ? S.cull_enabled != 0 : S.m_param[m * kMemberParams + 1] != 0.0;
    return cull_flag && on && finite3(o) && finite3(d) && d.x * d.x + d.y * d.y + d.z * d.z <= 1.0 + 1e-6;
}

__device__ __forceinline__ CullRay make_cull_ray(const DScene& S, int m, const V3& o, const V3& d) {
    CullRay c;
    double ca = S.cull_a, ch = S.cull_h, cb = S.cull_b, cc = S.cull_coord, cr = S.cull_radius;
    double c0 = S.cull_center[0], c1 = S.cull_center[1], c2 = S.cull_center[2];
    if (m >= 0) {
        const double* p = S.m_param + m * kMemberParams;
        ca = p[2]; ch = p[3]; cb = p[4]; cc = p[5]; cr = p[6]; c0 = p[7]; c1 = p[8]; c2 = p[9];
    }
    // upper bounds in FP32, every step rounded up (two FP64 square roots cost
    // more than the rest of a query's start)
    const float cx = __double2float_ru(fabs(o.x - c0)), cy = __double2float_ru(fabs(o.y - c1)),
                cz = __double2float_ru(fabs(o.z - c2));
    const float ax = __double2float_ru(fabs(o.x)), ay = __double2float_ru(fabs(o.y)), az = __double2float_ru(fabs(o.z));
    const float L = __fadd_ru(__fsqrt_ru(__fmaf_ru(cx, cx, __fmaf_ru(cy, cy, __fmul_ru(cz, cz)))), __double2float_ru(cr));
    const float on = __fsqrt_ru(__fmaf_ru(ax, ax, __fmaf_ru(ay, ay, __fmul_ru(az, az))));
    const float delta = __fmaf_ru(__double2float_ru(ca), __fadd_ru(L, __double2float_ru(ch)),
                                  __fmul_ru(__double2float_ru(cb), __fadd_ru(__fadd_ru(L, on), __double2float_ru(cc))));
    c.ox = static_cast<float>(o.x);
    c.oy = static_cast<float>(o.y);
    c.oz = static_cast<float>(o.z);
    c.ix = 1.0f / static_cast<float>(d.x);
    c.iy = 1.0f / static_cast<float>(d.y);
    c.iz = 1.0f / static_cast<float>(d.z);
    c.delta = __fmul_ru(delta, 1.0001f);
    return c;
}

// FP32 slab test of the ray [0, inf) against a box inflated by c.delta.
// Conservative: a triangle inside the box that the exact FP64 test accepts
// always passes (the inflation bounds both roundings); only work is skipped.
// Boxes are 6 floats on a 24-byte stride from a 16-byte aligned array
// (checked at upload): read as three 8-byte loads.
__device__ __forceinline__ bool cull_box(const float2& b01, const float2& b23, const float2& b45, const CullRay& c) {
    float t1 = (b01.x - c.delta - c.ox) * c.ix, t2 = (b23.y + c.delta - c.ox) * c.ix;
    float tmin = fmaxf(0.0f, fminf(t1, t2)), tmax = fmaxf(t1, t2);
    t1 = (b01.y - c.delta - c.oy) * c.iy; t2 = (b45.x + c.delta - c.oy) * c.iy;
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    t1 = (b23.x - c.delta - c.oz) * c.iz; t2 = (b45.y + c.delta - c.oz) * c.iz;
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    return tmin <= tmax;
}

__device__ __forceinline__ bool cull_box(const float* __restrict__ b, const CullRay& c) {
    return cull_box(*reinterpret_cast<const float2*>(b), *reinterpret_cast<const float2*>(b + 2),
                    *reinterpret_cast<const float2*>(b + 4), c);
}

// One leaf slot's record (DScene::leaf_rec).
struct LeafRec {
    float4 a, b;   // min xyz, max x | max yz, sub, object
    __device__ __forceinline__ int sub() const { return __float_as_int(b.z); }
    __device__ __forceinline__ int obj() const { return __float_as_int(b.w); }
};

__device__ __forceinline__ LeafRec load_leaf(const DScene& S, int slot) {
    LeafRec r;
    r.a = S.leaf_rec[2LL * slot];
    r.b = S.leaf_rec[2LL * slot + 1];
    return r;
}

// cull_box against a leaf record's box: a patch whose box fails has no block,
// cell or triangle that passes (the box is their union), so stage 1 misses.
// About two thirds of the patches of a visited leaf end here, for one box
// test and two 16-byte loads instead of 16 block boxes.
__device__ __forceinline__ bool cull_leaf(const LeafRec& r, const CullRay& c) {
    float t1 = (r.a.x - c.delta - c.ox) * c.ix, t2 = (r.a.w + c.delta - c.ox) * c.ix;
    float tmin = fmaxf(0.0f, fminf(t1, t2)), tmax = fmaxf(t1, t2);
    t1 = (r.a.y - c.delta - c.oy) * c.iy; t2 = (r.b.x + c.delta - c.oy) * c.iy;
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    t1 = (r.a.z - c.delta - c.oz) * c.iz; t2 = (r.b.y + c.delta - c.oz) * c.iz;
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    return tmin <= tmax;
}

// The n-th (from 0) set bit of m, which has more than n.
__device__ __forceinline__ int nth_bit(unsigned m, int n) {
    for (int k = 0; k < n; ++k) m &= m - 1u;
    return __ffs(m) - 1;
}

// FP32 BVH node test that reproduces ray_box_exact's decision or defers it.
//
// ray_box_exact(o, 1/d, box, best_t) passes exactly when, over the three
// axes, tmin = max(lo_a) <= tmax = min(hi_a), tmin <= best_t and tmax >= 0,
// where lo_a / hi_a are the FP64 slab times fl(fl(b - o) * fl(1/d)) of the
// near / far face (its early exit and swap give that; every t is finite for
// finite o and 1/d).  In FP32, with b32 = fl32(b), o32 = fl32(o), i32 =
// fl32(1 / fl32(d)) and p32 = fl32(-o32 * i32), each face's time is one
// fused multiply-add, fl32(b32 * i32 + p32).  It differs from the FP64 one by
// at most (5.01 * 2^-24 + 3 * 2^-53) (|b| + |o|) |1/d| plus underflow terms
// below 2^-120 (in units of 2^-24 |1/d|: roundings of b 1, of o 1, of d and
// the division 2 for each of b and o, of p 1, of the sum 1); e (make_node_ray)
// bounds that with 2^-21 (B_a + |o32_a|) |i32_a| for the largest axis, B_a
// bounding every node coordinate on axis a.  So the FP64 tmin lies within e of
// the FP32 one and likewise tmax, and the test decides wherever those intervals
// decide (directed rounding on the sums): 1 = passes, 0 = fails, -1 =
// undecided (run ray_box_exact).
struct NodeRay {
    float ix, iy, iz, px, py, pz;   // 1/d, -o/d
    float e, e2;                    // margin, and 2 e rounded up
    float best_hi, best_lo;         // best_t + e rounded up, best_t - e rounded down
    __device__ __forceinline__ void set_best(double best_t) {
        best_hi = __fadd_ru(__double2float_ru(best_t), e);
        best_lo = __fsub_rd(__double2float_rd(best_t), e);
    }
};

__device__ __forceinline__ int node_box_f32(float x0, float y0, float z0, float x1, float y1, float z1, const NodeRay& r) {
    float t1 = fmaf(x0, r.ix, r.px), t2 = fmaf(x1, r.ix, r.px);
    float tmin = fminf(t1, t2), tmax = fmaxf(t1, t2);
    t1 = fmaf(y0, r.iy, r.py); t2 = fmaf(y1, r.iy, r.py);
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    t1 = fmaf(z0, r.iz, r.pz); t2 = fmaf(z1, r.iz, r.pz);
    tmin = fmaxf(tmin, fminf(t1, t2)); tmax = fminf(tmax, fmaxf(t1, t2));
    if (tmin > __fadd_ru(tmax, r.e2) || tmax < -r.e || tmin > r.best_hi) return 0;
    if (tmin <= __fsub_rd(tmax, r.e2) && tmax >= r.e && tmin <= r.best_lo) return 1;
    return -1;
}

// A box of 6 floats (min xyz, max xyz), 8-byte aligned: three 8-byte loads.
__device__ __forceinline__ int node_box_f32(const float* __restrict__ b, const NodeRay& r) {
    const float2 b01 = *reinterpret_cast<const float2*>(b);
    const float2 b23 = *reinterpret_cast<const float2*>(b + 2);
    const float2 b45 = *reinterpret_cast<const float2*>(b + 4);
    return node_box_f32(b01.x, b01.y, b23.x, b23.y, b45.x, b45.y, r);
}

// The FP32 node test's ray (false: its values lie outside the range the bound
// covers, and its node tests stay FP64).  The limits keep every FP32 time below
// 2^81 and 1/d normal; the 2^-100 floor covers the underflow terms.  best_t is
// infinite.
__device__ __forceinline__ bool make_node_ray(const DScene& S, const CullRay& c, NodeRay& r) {
    const float o[3] = { c.ox, c.oy, c.oz }, iv[3] = { c.ix, c.iy, c.iz };
    float m = 0x1p-100f;
    bool ok = S.node_f32_ok != 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float ai = fabsf(iv[a]), ao = fabsf(o[a]);
        ok = ok && ai >= 0x1p-40f && ai <= 0x1p40f && ao <= 0x1p40f;
        m = fmaxf(m, __fmul_ru(__fadd_ru(S.node_bound[a], ao), ai) * 0x1p-21f);
    }
    r.ix = c.ix; r.iy = c.iy; r.iz = c.iz;
    r.px = -c.ox * c.ix; r.py = -c.oy * c.iy; r.pz = -c.oz * c.iz;
    r.e = m;
    r.e2 = 2.0f * m;
    r.best_hi = r.best_lo = CUDART_INF_F;
    return ok;
}

// Stage-1 winner bookkeeping.  key = ((cell * 3 + sign) * 2 + triangle) is
// the position of a test in the reference's loop order (i, j, sign 0/+1/-1,
// triangle); the reference keeps the first strictly smaller t, i.e. the
// smallest (t, key) pair, which is what this keeps in any visiting order.
struct Stage1 {
    bool have = false;
    double t = 0.0;
    int key = 0;
    __device__ __forceinline__ void consider(double tc, int kc) {
        if (!have || tc < t || (tc == t && kc < key)) { have = true; t = tc; key = kc; }
    }
};

// The six Moller-Trumbore tests of coarse cell (i, j): signs 0, +1, -1 of
// the cell's sagitta along its normal, triangles (q00,q10,q11), (q00,q11,q01).
__device__ __forceinline__ void stage1_cell(const double* __restrict__ X, const double* __restrict__ CC, int n,
                                            int i, int j, const V3& o, const V3& d, Stage1& best) {
    const int nc = n - 1;
    const double* r0 = X + static_cast<long long>(i * n + j) * 3;
    const double* r1 = r0 + 3 * n;
    const V3 p00 = load3(r0), p01 = load3(r0 + 3), p10 = load3(r1), p11 = load3(r1 + 3);
    const double* c = CC + static_cast<long long>(i * nc + j) * 4;
    const V3 cn = v3(c[0], c[1], c[2]);
    const double s = c[3];
    const int base = (i * nc + j) * 6;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double sg = (k == 0) ? 0.0 : ((k == 1) ? 1.0 : -1.0);
        const double dd = sg * s;
        const V3 q00 = v3(p00.x + cn.x * dd, p00.y + cn.y * dd, p00.z + cn.z * dd);
        const V3 q10 = v3(p10.x + cn.x * dd, p10.y + cn.y * dd, p10.z + cn.z * dd);
        const V3 q01 = v3(p01.x + cn.x * dd, p01.y + cn.y * dd, p01.z + cn.z * dd);
        const V3 q11 = v3(p11.x + cn.x * dd, p11.y + cn.y * dd, p11.z + cn.z * dd);
        double t;
        if (mt_exact(o, d, q00, q10, q11, t)) best.consider(t, base + 2 * k);
        if (mt_exact(o, d, q00, q11, q01, t)) best.consider(t, base + 2 * k + 1);
    }
}

// SurfacePatch::intersect stage 1: the winning (t, key) over the coarse
// triangulation (all cells, or only cells whose inflated box the ray crosses).
template <class Ctr>
__device__ __forceinline__ Stage1 patch_stage1(const DScene& S, int pidx, const V3& o, const V3& d, bool use_cull,
                                               const CullRay& cr, Ctr& ctr) {
    const int n = S.coarse_n, nc = n - 1;
    const double* X = S.c_xyz + static_cast<long long>(pidx) * n * n * 3;
    const double* CC = S.c_cell + static_cast<long long>(pidx) * nc * nc * 4;
    Stage1 best;
    ++ctr.patch_tests;
    if (use_cull) {
        const int B = S.block_cells, NB = S.n_blocks_side;
        const float* BB = S.c_block_box + static_cast<long long>(pidx) * NB * NB * 6;
        const float* CB = S.c_cell_box + static_cast<long long>(pidx) * nc * nc * 6;
        for (int bi = 0; bi < NB; ++bi) {
            for (int bj = 0; bj < NB; ++bj) {
                ++ctr.cell_tests;
                if (!cull_box(BB + (bi * NB + bj) * 6, cr)) continue;
                const int i1 = min(nc, (bi + 1) * B), j1 = min(nc, (bj + 1) * B);
                for (int i = bi * B; i < i1; ++i) {
                    for (int j = bj * B; j < j1; ++j) {
                        ++ctr.cell_tests;
                        if (!cull_box(CB + (i * nc + j) * 6, cr)) continue;
                        ctr.tri_tests += 6;
                        stage1_cell(X, CC, n, i, j, o, d, best);
                    }
                }
            }
        }
    } else {
        for (int i = 0; i < nc; ++i)
            for (int j = 0; j < nc; ++j) stage1_cell(X, CC, n, i, j, o, d, best);
        ctr.tri_tests += 6LL * nc * nc;
    }
    return best;
}

// triangle_uv_centroid (SurfacePatch.hpp:499-510) of the stage-1 winner `key`.
__device__ __forceinline__ void key_to_uv(const DScene& S, int key, double& u0, double& v0) {
    const int nc = S.coarse_n - 1;
    const int cell = key / 6;
    const bool second = (key & 1) != 0;
    const int bi = cell / nc, bj = cell % nc;
    const double ui = S.coarse_uv[bi], ui1 = S.coarse_uv[bi + 1];
    const double vj = S.coarse_uv[bj], vj1 = S.coarse_uv[bj + 1];
    if (!second) { u0 = (ui + ui1 + ui1) / 3.0; v0 = (vj + vj + vj1) / 3.0; }
    else         { u0 = (ui + ui + ui1) / 3.0; v0 = (vj + vj1 + vj1) / 3.0; }
}

// SurfacePatch::intersect: stage 1, then Newton from the winning triangle's
// (u, v) centroid and its t.
template <class Ctr>
__device__ __forceinline__ int patch_intersect(const DScene& S, int pidx, const V3& o, const V3& d, bool use_cull,
                                               const CullRay& cr, QHit& h, Ctr& ctr) {
    const Stage1 best = patch_stage1(S, pidx, o, d, use_cull, cr, ctr);
    if (!best.have) return 0;
    double u0, v0;
    key_to_uv(S, best.key, u0, v0);
    long long it = 0;
    const int r = newton_exact(S, pidx, o, d, u0, v0, best.t, h, it);
    ctr.newton_iters += it;
    return r;
}

// Triangle::intersect (Triangle.hpp:26-28): Moller-Trumbore, point o + t d,
// normal normalize(e1 x e2).
template <class Ctr>
__device__ __forceinline__ int triangle_intersect(const DScene& S, int sub, const V3& o, const V3& d, QHit& h,
                                                  Ctr& ctr) {
    h.err = 0;
    h.ev0 = 0.0;
    h.ev1 = 0.0;
    const double* v = S.tri + static_cast<long long>(sub) * 9;
    const V3 v0 = load3(v), v1 = load3(v + 3), v2 = load3(v + 6);
    double t, u, w;
    ++ctr.tri_tests;
    if (!mt_full(o, d, v0, v1, v2, t, u, w)) return 0;
    h.t = t;
    h.p = v3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
    h.n = vnormalize(vcross(vsub(v1, v0), vsub(v2, v0)));
    h.u = u;
    h.v = w;
    return 1;
}

// ScatObject::intersect for object `obj`: 1 hit, 0 miss (h.err set on a
// Newton failure).
template <class Ctr>
__device__ __forceinline__ int object_intersect(const DScene& S, int obj, const V3& o, const V3& d, bool use_cull,
                                                const CullRay& cr, QHit& h, Ctr& ctr) {
    h.err = 0;
    h.ev0 = 0.0;
    h.ev1 = 0.0;
    const int sub = S.obj_sub[obj];
    if (S.obj_kind[obj] == BBRT_OBJ_PATCH) return patch_intersect(S, sub, o, d, use_cull, cr, h, ctr);
    return triangle_intersect(S, sub, o, d, h, ctr);
}

// BVH::intersect with a 64-entry stack.  Returns the closest hit (obj >= 0),
// a miss (obj < 0, err 0), or the first Newton failure met (err != 0).
// off_patch_miss (learned form): a Newton root outside its patch is a miss.
// PATCHES false: a scene of triangles only (without stage 1 and the Newton solve
// a query kernel needs 96 registers and spills none).
template <bool PATCHES = true, class Ctr>
__device__ QHit bvh_query(const DScene& S, const V3& o, const V3& d, int cull_flag, Ctr& ctr,
                          bool off_patch_miss = false, int member = -1) {
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
        ++ctr.node_tests;
        if (!ray_box_exact(o, inv, S.node_box + 6LL * idx, best_t)) continue;
        const int* link = S.node_link + 4LL * idx;
        if (link[1] < 0) {
            const int start = link[0], count = link[2];
            for (int k = 0; k < count; ++k) {
                const LeafRec rec = load_leaf(S, start + k);
                const int obj = rec.obj();
                if (PATCHES && use_cull && rec.sub() >= 0 && !cull_leaf(rec, cr)) {
                    ++ctr.patch_tests;
                    ++ctr.cell_tests;
                    continue;
                }
                QHit h;
                int r;
                if constexpr (PATCHES) r = object_intersect(S, obj, o, d, use_cull, cr, h, ctr);
                else r = triangle_intersect(S, ~rec.sub(), o, d, h, ctr);
                if (off_patch_miss && h.err == BBRT_RAY_NEWTON_DOMAIN) {
                    ++ctr.off_patch;
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

__device__ __forceinline__ void warp_add(long long* dst, long long v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(reinterpret_cast<unsigned long long*>(dst), static_cast<unsigned long long>(v));
}

// ---- the bounce loop (RayTracingDriver::trace_ray) as per-ray state steps ----

// Registers of one ray between queries.
struct RayCtx {
    V3 o, d;
    int member;      // scene-set member of the ray, -1 for a single scene
    int bounces;
    int status;      // final status once set; -1 while the ray is running
    int err_obj;
    double ev0, ev1;
};

__device__ __forceinline__ void init_outputs(const TraceArgs& A, long long i) {
    if (A.ray_work) for (int k = 0; k < 4; ++k) A.ray_work[4 * i + k] = 0;
    const int K = A.record;
    for (int k = 0; k < K; ++k) {
        if (A.hit_object) A.hit_object[i * K + k] = -1;
        if (A.hit_point) { double* p = A.hit_point + (i * K + k) * 3; p[0] = 0.0; p[1] = 0.0; p[2] = 0.0; }
        if (A.hit_uv) { double* p = A.hit_uv + (i * K + k) * 2; p[0] = 0.0; p[1] = 0.0; }
    }
}

// Start of trace_ray: zero-length check, normalisation (RayTracingDriver.hpp:174-184).
__device__ __forceinline__ RayCtx start_ray(const TraceArgs& A, long long i) {
    RayCtx r;
    r.o = load3(A.origins + 3 * i);
    r.member = A.ray_member ? A.ray_member[i] : -1;
    const V3 dir_in = load3(A.dirs + 3 * i);
    r.d = v3(0.0, 0.0, 0.0);
    r.bounces = 0;
    r.status = -1;
    r.err_obj = -1;
    r.ev0 = r.ev1 = 0.0;
    const double len2 = dir_in.x * dir_in.x + dir_in.y * dir_in.y + dir_in.z * dir_in.z;
    if (len2 < 1e-300) {
        r.status = BBRT_RAY_BAD_DIR;
    } else {
        const double len = sqrt(dir_in.x * dir_in.x + dir_in.y * dir_in.y + dir_in.z * dir_in.z);
        r.d = v3(dir_in.x / len, dir_in.y / len, dir_in.z / len);
    }
    return r;
}

// A single query's ray: as given.
__device__ __forceinline__ RayCtx start_query(const TraceArgs& A, long long i) {
    RayCtx r;
    r.o = load3(A.origins + 3 * i);
    r.d = load3(A.dirs + 3 * i);
    r.member = -1;
    r.bounces = 0;
    r.status = -1;
    r.err_obj = -1;
    r.ev0 = r.ev1 = 0.0;
    return r;
}

// The last recorded point of a ray, kept in the caller's array from bounce to
// bounce rather than in the ray's state.
__device__ __forceinline__ void put_end(const TraceArgs& A, long long i, const V3& p) {
    if (!A.end_point) return;
    double* e = A.end_point + 3 * i;
    e[0] = p.x; e[1] = p.y; e[2] = p.z;
}

// One bounce of trace_ray given the query result h (RayTracingDriver.hpp:187-237).
// Returns true when the ray goes on to another query.
__device__ __forceinline__ bool step_ray(const DScene& S, const TraceArgs& A, long long i, RayCtx& r, const QHit& h,
                                        bool write = true) {
    if (h.err) {
        r.status = h.err;
        r.err_obj = h.obj;
        r.ev0 = h.ev0;
        r.ev1 = h.ev1;
        return false;
    }
    if (h.obj < 0) {
        r.status = BBRT_RAY_ESCAPED;
        const double diag = scene_diag(S, r.member);
        if (write) put_end(A, i, v3(r.o.x + r.d.x * diag, r.o.y + r.d.y * diag, r.o.z + r.d.z * diag));
        return false;
    }
    if (vdot(r.d, h.n) > S.backface_tol) { r.status = BBRT_RAY_WENT_INSIDE; return false; }
    const int K = A.record;
    if (write && r.bounces < K) {
        if (A.hit_object) A.hit_object[i * K + r.bounces] = h.obj;
        if (A.hit_point) { double* p = A.hit_point + (i * K + r.bounces) * 3; p[0] = h.p.x; p[1] = h.p.y; p[2] = h.p.z; }
        if (A.hit_uv) { double* p = A.hit_uv + (i * K + r.bounces) * 2; p[0] = h.u; p[1] = h.v; }
    }
    if (write && A.hit_counts && r.bounces >= A.count_from) atomicAdd(A.hit_counts + h.obj, 1ULL);
    ++r.bounces;
    if (write) put_end(A, i, h.p);
    const V3 d = r.d;
    const double dn = d.x * h.n.x + d.y * h.n.y + d.z * h.n.z;
    r.d = v3(d.x - 2.0 * dn * h.n.x, d.y - 2.0 * dn * h.n.y, d.z - 2.0 * dn * h.n.z);
    const double eps = smax(S.eps_factor * scene_diag(S, r.member), S.sag_factor * S.obj_pad[h.obj]);
    r.o = v3(h.p.x + r.d.x * eps, h.p.y + r.d.y * eps, h.p.z + r.d.z * eps);
    return true;
}

__device__ __forceinline__ void finish_ray(const TraceArgs& A, long long i, const RayCtx& r) {
    if (A.status) A.status[i] = r.status;
    if (A.bounce_count) A.bounce_count[i] = r.bounces;
    if (A.exit_dir) { double* p = A.exit_dir + 3 * i; p[0] = r.d.x; p[1] = r.d.y; p[2] = r.d.z; }
    // escaped rays and rays with a bounce have their end point already
    if (r.bounces == 0 && r.status != BBRT_RAY_ESCAPED) put_end(A, i, load3(A.origins + 3 * i));
    if (A.err_object) A.err_object[i] = r.err_obj;
    if (A.err_value) { A.err_value[2 * i] = r.ev0; A.err_value[2 * i + 1] = r.ev1; }
}

// Runs the bounce loop of one ray to the end with inline queries.
template <class Ctr>
__device__ __forceinline__ void run_ray(const DScene& S, const TraceArgs& A, long long i, RayCtx& r, Ctr& ctr,
                                        long long& queries) {
    while (r.status < 0) {
        if (r.bounces >= A.max_bounces) { r.status = BBRT_RAY_MAX_BOUNCES; break; }
        ++queries;
        const QHit h = bvh_query(S, r.o, r.d, A.cull, ctr, A.off_patch_miss != 0, r.member);
        if (!step_ray(S, A, i, r, h)) break;
    }
}

// Adds one thread's work counters for ray i to the optional per-ray profile
// (a ray is owned by one thread at a time, so no atomics are needed).
template <class Ctr>
__device__ __forceinline__ void add_ray_work(const TraceArgs& A, long long i, const Ctr& c) {
    if constexpr (!Ctr::kOn) return;
    if (!A.ray_work || i < 0) return;
    long long* w = A.ray_work + 4 * i;
    w[0] += c.node_tests;
    w[1] += c.cell_tests;
    w[2] += c.tri_tests;
    w[3] += c.newton_iters;
}

template <bool ON>
struct RayTallyT {
    long long bounces = 0, queries = 0;
    long long hist[BBRT_RAY_STATUS_COUNT] = { 0, 0, 0, 0, 0, 0, 0, 0 };
};
template <>
struct RayTallyT<false> {
    NoCount bounces, queries;
    NoCount hist[BBRT_RAY_STATUS_COUNT];
};
using RayTally = RayTallyT<true>;

template <class Ctr, class Tally>
__device__ __forceinline__ void flush_stats(const TraceArgs& A, const Ctr& ctr, const Tally& t, bool tail = false) {
    if constexpr (!Ctr::kOn) return;
    if (!A.stats) return;
    if (tail) {
        long long rays = 0;
#pragma unroll
        for (int k = 0; k < BBRT_RAY_STATUS_COUNT; ++k) rays += t.hist[k];
        warp_add(A.stats + ST_TAIL_NODE_TESTS, ctr.node_tests);
        warp_add(A.stats + ST_TAIL_CELL_TESTS, ctr.cell_tests);
        warp_add(A.stats + ST_TAIL_TRI_TESTS, ctr.tri_tests);
        warp_add(A.stats + ST_TAIL_NEWTON_ITERS, ctr.newton_iters);
        warp_add(A.stats + ST_TAIL_RAYS, rays);
    }
    warp_add(A.stats + ST_BOUNCES, t.bounces);
    warp_add(A.stats + ST_QUERIES, t.queries);
    warp_add(A.stats + ST_NODE_TESTS, ctr.node_tests);
    warp_add(A.stats + ST_PATCH_TESTS, ctr.patch_tests);
    warp_add(A.stats + ST_CELL_TESTS, ctr.cell_tests);
    warp_add(A.stats + ST_TRI_TESTS, ctr.tri_tests);
    warp_add(A.stats + ST_NEWTON_ITERS, ctr.newton_iters);
    warp_add(A.stats + ST_OFF_PATCH, ctr.off_patch);
    warp_add(A.stats + ST_NODE_F64, ctr.node_f64);
#pragma unroll
    for (int k = 0; k < BBRT_RAY_STATUS_COUNT; ++k) warp_add(A.stats + ST_HIST0 + k, t.hist[k]);
}

// A query's outcome as the caller's record.
__device__ __forceinline__ void write_hit(bbrt_hit* out, const QHit& r) {
    bbrt_hit w;
    w.t = 0.0;
    for (int k = 0; k < 3; ++k) { w.point[k] = 0.0; w.normal[k] = 0.0; }
    w.uv[0] = w.uv[1] = 0.0;
    w.object = -1;
    w.status = 0;
    w.err_object = -1;
    w.pad_ = 0;
    w.err_value[0] = w.err_value[1] = 0.0;
    if (r.err) {
        w.status = r.err;
        w.err_object = r.obj;
        w.err_value[0] = r.ev0;
        w.err_value[1] = r.ev1;
    } else if (r.obj >= 0) {
        w.t = r.t;
        w.point[0] = r.p.x; w.point[1] = r.p.y; w.point[2] = r.p.z;
        w.normal[0] = r.n.x; w.normal[1] = r.n.y; w.normal[2] = r.n.z;
        w.uv[0] = r.u; w.uv[1] = r.v;
        w.object = r.obj;
    }
    *out = w;
}

// ---- wavefront form: advance rays until they need a Newton solve ----------

__device__ __forceinline__ void save_ray(const WaveArgs& W, long long i, const RayCtx& r, int nres) {
    double* o = W.o + 3 * i;
    double* d = W.d + 3 * i;
    o[0] = r.o.x; o[1] = r.o.y; o[2] = r.o.z;
    d[0] = r.d.x; d[1] = r.d.y; d[2] = r.d.z;
    W.bounces[i] = r.bounces;
    W.nres[i] = nres;
}

__device__ __forceinline__ RayCtx load_ray(const TraceArgs& A, const WaveArgs& W, long long i, int& nres) {
    RayCtx r;
    r.member = A.ray_member ? A.ray_member[i] : -1;
    r.o = load3(W.o + 3 * i);
    r.d = load3(W.d + 3 * i);
    r.bounces = W.bounces[i];
    r.status = -1;
    r.err_obj = -1;
    r.ev0 = r.ev1 = 0.0;
    nres = W.nres ? W.nres[i] : 0;
    return r;
}

// Appends one training sample (learned guess) when recording is on.
__device__ __forceinline__ void record_sample(const TraceArgs& A, int label, const V3& o, const V3& d, int pidx,
                                              double u, double v, double t) {
    const unsigned long long k = atomicAdd(A.sample_count + label, 1ULL);
    const long long cap = label ? A.sample_cap_pos : A.sample_cap_neg;
    if (static_cast<long long>(k) >= cap) return;
    GuessSample* s = A.samples + (label ? 0 : A.sample_cap_pos) + k;
    s->o[0] = o.x; s->o[1] = o.y; s->o[2] = o.z;
    s->d[0] = d.x; s->d[1] = d.y; s->d[2] = d.z;
    s->u = u; s->v = v; s->t = t;
    s->patch = pidx;
    s->label = label;
}

// One of the six Moller-Trumbore tests of cell (i, j): step = 2 * sign + triangle,
// sign order 0, +1, -1 of the sagitta along the cell normal, triangles
// (q00,q10,q11) then (q00,q11,q01) — the order and arithmetic of stage1_cell.
__device__ __forceinline__ void stage1_tri(const double* __restrict__ X, const double* __restrict__ CC, int n, int i,
                                           int j, int step, const V3& o, const V3& d, Stage1& best) {
    const int nc = n - 1;
    const double* r0 = X + static_cast<long long>(i * n + j) * 3;
    const double* r1 = r0 + 3 * n;
    // cell normal and sagitta: 4 doubles on a 32-byte stride (16-byte loads)
    const double* c = CC + static_cast<long long>(i * nc + j) * 4;
    const double2 c01 = *reinterpret_cast<const double2*>(c);
    const double2 c23 = *reinterpret_cast<const double2*>(c + 2);
    const V3 cn = v3(c01.x, c01.y, c23.x);
    const int k = step >> 1;
    const double sg = (k == 0) ? 0.0 : ((k == 1) ? 1.0 : -1.0);
    const double dd = sg * c23.y;
    const V3 p00 = load3(r0), p11 = load3(r1 + 3);
    const V3 pm = (step & 1) ? load3(r0 + 3) : load3(r1);   // p01 for the second triangle, p10 for the first
    const V3 q00 = v3(p00.x + cn.x * dd, p00.y + cn.y * dd, p00.z + cn.z * dd);
    const V3 q11 = v3(p11.x + cn.x * dd, p11.y + cn.y * dd, p11.z + cn.z * dd);
    const V3 qm = v3(pm.x + cn.x * dd, pm.y + cn.y * dd, pm.z + cn.z * dd);
    double t;
    const bool hit = (step & 1) ? mt_exact(o, d, q00, q11, qm, t) : mt_exact(o, d, q00, qm, q11, t);
    if (hit) best.consider(t, (i * nc + j) * 6 + step);
}

// One of the two triangles of cell (i, j) (second: q00, q11, q01) at all three
// signs, in stage1_tri's order and arithmetic, its corners loaded once.
__device__ __forceinline__ void stage1_tri3(const double* __restrict__ X, const double* __restrict__ CC, int n, int i,
                                            int j, bool second, const V3& o, const V3& d, Stage1& best) {
    const int nc = n - 1;
    const double* r0 = X + static_cast<long long>(i * n + j) * 3;
    const double* r1 = r0 + 3 * n;
    const double* c = CC + static_cast<long long>(i * nc + j) * 4;
    const double2 c01 = *reinterpret_cast<const double2*>(c);
    const double2 c23 = *reinterpret_cast<const double2*>(c + 2);
    const V3 cn = v3(c01.x, c01.y, c23.x);
    // the triangle's second and third corner: (q10, q11), or (q11, q01)
    const V3 p0 = load3(r0), p1 = load3(second ? r1 + 3 : r1), p2 = load3(second ? r0 + 3 : r1 + 3);
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const double sg = (k == 0) ? 0.0 : ((k == 1) ? 1.0 : -1.0);
        const double dd = sg * c23.y;
        const V3 q0 = v3(p0.x + cn.x * dd, p0.y + cn.y * dd, p0.z + cn.z * dd);
        const V3 q1 = v3(p1.x + cn.x * dd, p1.y + cn.y * dd, p1.z + cn.z * dd);
        const V3 q2 = v3(p2.x + cn.x * dd, p2.y + cn.y * dd, p2.z + cn.z * dd);
        double t;
        if (mt_exact(o, d, q0, q1, q2, t)) best.consider(t, (i * nc + j) * 6 + 2 * k + (second ? 1 : 0));
    }
}

// ---- warp-cooperative stage 1 (used by k_advance and the warp-per-ray kernels) ----

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ void warp_min_stage1(Stage1& s) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int oh = __shfl_xor_sync(kFull, s.have ? 1 : 0, off);
        const double ot = __shfl_xor_sync(kFull, s.t, off);
        const int ok = __shfl_xor_sync(kFull, s.key, off);
        if (oh) s.consider(ot, ok);
    }
}

// Lane `lane` runs the `k`-th of the six triangle tests of each passing cell in
// `cm` (cells enumerated by the set bits of cm, offsets into (ci0, cj0) grid of
// width w), 32 tests at a time.
__device__ __forceinline__ void warp_cell_tris(const double* X, const double* CC, int n, unsigned cm, int base_i,
                                               int base_j, int w, int c0, const V3& o, const V3& d, int lane,
                                               Stage1& best) {
    const int total = __popc(cm) * 6;
    for (int p0 = 0; p0 < total; p0 += 32) {
        const int p = p0 + lane;
        if (p < total) {
            const int c = c0 + nth_bit(cm, p / 6);
            stage1_tri(X, CC, n, base_i + c / w, base_j + c % w, p % 6, o, d, best);
        }
    }
}

template <class Ctr>
__device__ Stage1 warp_patch_stage1(const DScene& S, int pidx, const V3& o, const V3& d, bool use_cull,
                                    const CullRay& cr, int lane, Ctr& ctr) {
    const int n = S.coarse_n, nc = n - 1;
    const double* X = S.c_xyz + static_cast<long long>(pidx) * n * n * 3;
    const double* CC = S.c_cell + static_cast<long long>(pidx) * nc * nc * 4;
    Stage1 best;
    if (lane == 0) ++ctr.patch_tests;
    if (!(finite3(o) && finite3(d))) {
        // ordered loop on every lane (same result everywhere)
        CountersT<false> dummy;
        best = patch_stage1(S, pidx, o, d, false, cr, dummy);
        if (lane == 0) ctr.tri_tests += 6LL * nc * nc;
        return best;
    }
    if (use_cull) {
        const int B = S.block_cells, NB = S.n_blocks_side, NB2 = NB * NB;
        const float* BB = S.c_block_box + static_cast<long long>(pidx) * NB2 * 6;
        const float* CB = S.c_cell_box + static_cast<long long>(pidx) * nc * nc * 6;
        for (int b0 = 0; b0 < NB2; b0 += 32) {
            const int b = b0 + lane;
            unsigned bm = __ballot_sync(kFull, b < NB2 && cull_box(BB + b * 6, cr));
            if (lane == 0) ctr.cell_tests += min(32, NB2 - b0);
            while (bm) {
                const int bl = __ffs(bm) - 1;
                bm &= bm - 1;
                const int bi = (b0 + bl) / NB, bj = (b0 + bl) % NB;
                const int i0 = bi * B, j0 = bj * B;
                const int h = min(nc, i0 + B) - i0, w = min(nc, j0 + B) - j0;
                for (int c0 = 0; c0 < h * w; c0 += 32) {
                    const int c = c0 + lane;
                    const unsigned cm = __ballot_sync(kFull, c < h * w && cull_box(CB + ((i0 + c / w) * nc + j0 + c % w) * 6, cr));
                    if (lane == 0) { ctr.cell_tests += min(32, h * w - c0); ctr.tri_tests += 6 * __popc(cm); }
                    warp_cell_tris(X, CC, n, cm, i0, j0, w, c0, o, d, lane, best);
                }
            }
        }
    } else {
        const int total = nc * nc * 6;
        for (int p = lane; p < total; p += 32) stage1_tri(X, CC, n, (p / 6) / nc, (p / 6) % nc, p % 6, o, d, best);
        if (lane == 0) ctr.tri_tests += total;
    }
    warp_min_stage1(best);
    return best;
}

}  // namespace bbrt
