// Device-side scene view and launch descriptors shared by the host C ABI
// (capi.cpp) and the kernels (*.cu).  Plain pointers into one scene's device
// allocation; passed to kernels by value.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

namespace bbrt {

struct GuessSample;

struct DScene {
    int n_objects = 0;
    int n_nodes = 0;
    int coarse_n = 0;               // coarse grid is coarse_n x coarse_n for every patch
    int newton_max_iters = 20;
    double newton_tol = 1e-3;
    double scene_diagonal = 0.0;
    double max_patch_sagitta = 0.0;
    double eps_factor = 1e-9;       // kSelfIntersectEpsilonFactor
    double sag_factor = 5.0;        // kSagittaClearanceFactor
    double backface_tol = 1e-9;     // kBackfaceHitTol

    // BVH nodes renumbered breadth-first (the top levels come first) with
    // explicit children; the tree and its child order are the reference's.
    const double* node_box = nullptr;      // [n_nodes][6]  min xyz, max xyz
    const int* node_link = nullptr;        // [n_nodes][4]  internal: left, right, 0, axis
                                           //               leaf:     start, -1, count, 0
    const int* leaf_objects = nullptr;
    // Leaf records, one per leaf slot (leaf_objects order), 32 bytes each as
    // two 16-byte halves: the object's stage-1 cull box (min xyz, max xyz:
    // the union of the patch's block boxes; -inf / +inf for a triangle or
    // without cull tables), then its patch index (or ~triangle index) and its
    // object index, both as int bits.
    const float4* leaf_rec = nullptr;
    // The tree's leaves for queries that look them up instead of walking
    // (ray_warp.cu), in depth-first (left before right) order, a scene set's
    // members one after the other:
    //   leaf_box  [n_leaves][6] FP64 box;  leaf_node [n_leaves] two float4: FP32
    //   box, first slot and slot count (int bits)
    //   leaf_rank [n_leaves][8] place in the depth-first order of a ray whose
    //   1/d is negative on the axes in the octant's bits
    //   cut_rec   the largest subtrees of at most 32 leaves, two float4 each:
    //   FP32 box, first leaf and leaf count; cut_box their FP64 boxes
    //   m_cut     first cut of each member ({0, count} for one scene)
    // leaf_lists = 0: not usable (a box beyond the FP32 test's range, or a tree
    // so deep that a walk could overflow its stack).
    int leaf_lists = 0;
    int node_f32 = 1;                      // 0: the warp-per-ray kernels test nodes in FP64 only
    const double* leaf_box = nullptr;
    const float4* leaf_node = nullptr;
    const int* leaf_rank = nullptr;
    const float4* cut_rec = nullptr;
    const double* cut_box = nullptr;
    const int* m_cut = nullptr;
    // The tree's internal nodes for k_advance, breadth-first: a record holds
    // both children, as four float4: their FP32 boxes (left, then right: 12
    // floats), then as int bits the left child's node index (the right one's
    // follows it), the children's references and the split axis.  A reference
    // is a record index, or ~leaf for a leaf (in leaf_node's order).
    // pair_node[r]: node index of record r; m_ref: reference of each tree's root.
    int n_pairs = 0;
    const float4* pair_rec = nullptr;
    const int* pair_node = nullptr;
    const int* m_ref = nullptr;
    int smem_pairs = 0;                    // records [0, smem_pairs) staged in shared memory
    // FP32 copies of the node boxes (nearest rounding) for the FP32 node
    // test, and per axis a bound on |coordinate| over every node box (FP32,
    // rounded up, at least 2^-60); node_f32_ok = 0 when a bound exceeds 2^40
    // (the test then stays FP64).
    const float* node_box32 = nullptr;     // [n_nodes][6]
    float node_bound[3] = { 0.0f, 0.0f, 0.0f };
    int node_f32_ok = 0;

    // objects
    const int* obj_kind = nullptr;         // BBRT_OBJ_*
    const int* obj_sub = nullptr;          // patch or triangle index
    const double* obj_pad = nullptr;       // self_intersect_padding

    // patches
    const int* p_dims = nullptr;           // [n_patches][2] imax, jmax
    const long long* p_node_off = nullptr; // un[imax] vn[jmax] uw[imax] vw[jmax]
    const long long* p_field_off = nullptr;// node-major, 12 doubles per node
    const double* p_nodes = nullptr;
    const double* p_fields = nullptr;
    const float* p_nodes32 = nullptr;      // FP32 copies (same offsets) for the FP32 Newton phase
    const float* p_fields32 = nullptr;
    int precision = 0;                     // BBRT_PREC_*
    int max_nodes = 0;                     // largest node count per axis over the patches
    const double* coarse_uv = nullptr;     // [coarse_n]
    const double* c_xyz = nullptr;         // [n_patches][coarse_n^2][3]
    const double* c_cell = nullptr;        // [n_patches][(coarse_n-1)^2][4] normal xyz, sagitta
    const float* c_cell_box = nullptr;     // [n_patches][(coarse_n-1)^2][6] cell AABB (cull)
    const float* c_block_box = nullptr;    // [n_patches][n_blocks][6] block AABB (cull)
    int block_cells = 4;                   // a block is block_cells x block_cells cells
    int n_blocks_side = 0;                 // blocks per side
    // Conservative inflation of the cull boxes for a ray with origin o:
    //   L     = |o - cull_center| + cull_radius   (bounds |o - v| for every vertex v)
    //   delta = cull_a * (L + cull_h) + cull_b * (L + |o| + cull_coord)
    // cull_a covers the FP64 Moller-Trumbore rounding (hits accepted up to that
    // far outside a triangle), cull_b the FP32 slab test's own rounding.
    int cull_enabled = 0;
    double cull_a = 0.0, cull_h = 0.0, cull_b = 0.0, cull_coord = 0.0;
    double cull_center[3] = { 0.0, 0.0, 0.0 };
    double cull_radius = 0.0;

    // Quadtree of a patch's cull boxes for k_stage1 (grids of at most 16 x 16
    // cells): kQuadNodes boxes a patch, 2 x 2, 4 x 4, 8 x 8 and 16 x 16 of them,
    // each level in Morton order (a node's four children side by side); a node
    // without cells has min > max.  Null for larger grids.
    const float* quad_box = nullptr;       // [n_patches][kQuadNodes][6]

    // triangles
    const double* tri = nullptr;           // [n_tri][9]

    // Several scenes traced as one (a scene set): the member scenes' objects,
    // patches and BVH trees live in the arrays above side by side; member m's
    // tree starts at node m_root[m], and its scale and cull constants are
    // m_param[m * kMemberParams + ...] (see kMemberParams).  n_members == 0
    // for a single scene, whose tree starts at node 0.
    int n_members = 0;
    const int* m_root = nullptr;
    const double* m_param = nullptr;
};

constexpr int kQuadNodes = 4 + 16 + 64 + 256;
// Per-member values of a scene set: scene diagonal, cull on (1) / off (0),
// cull_a, cull_h, cull_b, cull_coord, cull_radius, cull_center xyz.
constexpr int kMemberParams = 10;

// Counter slots of the per-launch statistics buffer (long long each).
enum StatSlot {
    ST_BOUNCES = 0, ST_QUERIES, ST_NODE_TESTS, ST_PATCH_TESTS, ST_CELL_TESTS, ST_TRI_TESTS,
    ST_NEWTON_ITERS, ST_NEWTON_ITERS_FP32, ST_HIST0,
    // share of the tail kernels (also included in the totals above)
    ST_TAIL_NODE_TESTS = ST_HIST0 + 8, ST_TAIL_CELL_TESTS, ST_TAIL_TRI_TESTS, ST_TAIL_NEWTON_ITERS, ST_TAIL_RAYS,
    // learned guess: Newton solves started from the network, and those that fell back to the triangle
    ST_GUESS_USED, ST_GUESS_FALLBACK,
    // learned form: patches whose Newton root lay outside the patch, taken as not hit
    ST_OFF_PATCH,
    // FP32 node test: node tests it left undecided (run in FP64)
    ST_NODE_F64,
    ST_COUNT
};

struct TraceArgs {
    const double* origins = nullptr;   // [n][3]
    const double* dirs = nullptr;      // [n][3]
    long long n = 0;
    int max_bounces = 0;
    int record = 0;                    // K
    int cull = 1;
    int* status = nullptr;
    int* bounce_count = nullptr;
    double* exit_dir = nullptr;
    double* end_point = nullptr;
    int* hit_object = nullptr;         // [n][K]
    double* hit_point = nullptr;       // [n][K][3]
    double* hit_uv = nullptr;          // [n][K][2]
    int* err_object = nullptr;
    double* err_value = nullptr;       // [n][2]
    long long* ray_work = nullptr;     // [n][4] node tests, box tests, MT tests, Newton iterations
    unsigned long long* hit_counts = nullptr;  // per object (plane source), may be null
    int count_from = 1;                // first bounce index that is counted
    long long* stats = nullptr;        // [ST_COUNT], may be null
    unsigned long long* work_counter = nullptr;  // persistent-launch ray counter (zeroed by host)
    // Training-sample recording (learned guess): converged Newton solves go to
    // samples[0, cap_pos), stage-1 misses to samples[cap_pos, cap_pos + cap_neg);
    // sample_count[1] / [0] count positives / negatives offered (may exceed the caps).
    GuessSample* samples = nullptr;
    unsigned long long* sample_count = nullptr;
    long long sample_cap_pos = 0, sample_cap_neg = 0;
    // Learned form: a patch whose Newton solve converges to a root outside
    // the patch's parameter domain (|u| or |v| > 1 + 1e-6) is taken as not
    // hit instead of failing the ray, unless the network placed a confident
    // hit well inside the patch (then the root is suspect and the failure
    // stands).  Off (0) in the plain and split forms, which keep the
    // reference's failure.
    int off_patch_miss = 0;
    // Scene set: the member scene of every ray ([n]); null for one scene.
    const int* ray_member = nullptr;
    // Single queries run as a round (rounds.cu, ray_warp.cu): bbrt_hit per ray,
    // directions as they are, nothing else written; null for a trace.
    void* query_out = nullptr;
};

// Network outputs (u, v, t, logit) that place a confident hit well inside
// the patch: they veto the learned form's off-patch miss.
__host__ __device__ inline bool guess_inside(const double* g, double min_logit) {
    return g != nullptr && g[3] > min_logit && fabs(g[0]) <= 0.95 && fabs(g[1]) <= 0.95;
}

// A patch query of the current bounce whose stage-1 winner needs Newton.
struct NewtonRequest {
    int ray;      // ray index
    int entry;    // slot in the ray's resolved list
    int obj;      // object index of the patch
    int key;      // stage-1 winner
    double t0;    // stage-1 t
};

// Resolved Newton results of a ray's current query: res_obj[ray][k] and
// res_data[ray][k][kResData] = t, point xyz, normal xyz, u, v, ev0, ev1.
constexpr int kResolved = 4;
constexpr int kResData = 11;

// Split rounds (rounds.cu): leaves a ray's query may list, slots a leaf may
// have, stage-1 hits and Newton results kept per ray.
constexpr int kSplitLeaves = 32, kSplitLeafSlots = 4, kSplitHits = 8, kSplitResults = 2;

// One stage-1 hit of a ray's query, in visiting order.
struct SplitHit {
    double t;
    int obj, leaf, key, pad;
};

// Round control of a graph-launched split round (its last k_stage1 block).
struct RoundControl {
    int on = 0;
    long long wave_tail = 0, max_rounds = 0;
    cudaGraphConditionalHandle loop = 0;
};

// Workspace of the wavefront trace (advance / Newton rounds).
struct WaveArgs {
    double* o = nullptr;       // [n][3] ray state between rounds
    double* d = nullptr;
    int* bounces = nullptr;
    int* nres = nullptr;
    int* res_obj = nullptr;    // [n][kResolved]
    int* res_err = nullptr;    // [n][kResolved]
    double* res_data = nullptr;  // [n][results][kResData]
    int results = kResolved;     // results per ray (kSplitResults in split rounds); a request's entry is
                                 // its result's slot, in split rounds with the hit's place << 1
    // Split rounds: a query's leaves in visiting order, its stage-1 hits, the
    // best result so far (hit << 1 | slot, -1 none), the rays that have leaves
    int* leaves = nullptr;       // [n][kSplitLeaves]
    int* n_leaves = nullptr;
    SplitHit* hits = nullptr;    // [n][kSplitHits]
    int* n_hits = nullptr;
    int* best = nullptr;
    int* listed = nullptr;
    const NewtonRequest* runnable = nullptr;   // previous round's requests (null: round 0, all rays)
    const int* order = nullptr;                // round 0 processing order (null: index order)
    long long n_runnable = 0;
    NewtonRequest* req = nullptr;              // this round's requests
    unsigned int* counters = nullptr;          // [0] requests of the round, [1] overflowed rays (cumulative),
                                               // [2] runnable rays fetched this round, [3] watchdog tripped
    int* overflow = nullptr;                   // rays whose query needs more than kResolved solves
    // Learned guess of this round's requests: guess[r] = (u, v, t, logit), or null.
    const double* guess = nullptr;
    const double* frame = nullptr;             // per-patch frames (size L at [12] of each 16)
    double guess_min_logit = 0.0;              // confidence needed to start Newton from the guess
    double guess_t_window = 0.5;               // accepted |t - t_stage1| in units of L
    // Traversal state of a query suspended for a Newton solve, so that the
    // next round resumes it instead of replaying it from the root:
    // qs_int[ray][kQsInt] = stack depth (-1: none saved), leaf slot, end of the
    // leaf's slots, best object, best resolved entry; qs_t[ray] = best t;
    // qs_stack[ray][kSaveStack].
    int* qs_int = nullptr;
    double* qs_t = nullptr;
    int* qs_stack = nullptr;
    int resume_queries = 1;
    int group_newton = 0;                      // Newton solves by 8-lane groups when the patches allow it
    // Graph-launched trace: the launch's item count (runnable rays, requests,
    // tail rays) is read from this device word instead of the host argument,
    // and the Newton kernel copies each request it solves to next_req (the
    // next round's runnable set); null in the host-driven trace.
    const unsigned int* count_dev = nullptr;
    NewtonRequest* next_req = nullptr;
    // k_advance stops (counters[3] set) once it has run this many SM cycles.
    long long watchdog_cycles = 1LL << 35;
    // k_advance and the warp-per-ray tail test BVH nodes in FP32
    // (node_box_f32), in FP64 only where the FP32 interval does not decide;
    // the visit sequence is unchanged.
    int node_f32 = 0;
    // k_advance: in a round with fewer rays than the grid's lanes, fewer
    // lanes of each warp take rays, spreading the round over every warp.
    int adapt_lanes = 0;
    // Rounds of at most this many Newton requests solve each with 8 lanes
    // (patches of at most 8 nodes per axis); 0: one request per thread always.
    long long newton_group_max = 0;
};

// Round counters of the wavefront trace in device memory: [0..3] as
// WaveArgs::counters; [4..7] are the round control of the graph-launched
// trace, written by k_wave_decide after each k_advance; [8..9] hand out the
// tail kernels' rays.  All start at zero for each trace.
constexpr int kWcNext = 4;     // requests solved this round, runnable next round (0: rounds end)
constexpr int kWcTail = 5;     // requests left to the tail kernel (the last, small round)
constexpr int kWcRounds = 6;   // rounds whose requests went to Newton
constexpr int kWcBound = 7;    // the round bound was reached
constexpr int kWcTailNext = 8; // next slot of the tail kernel (rays handed out one at a time)
constexpr int kWcOvfNext = 9;  // next slot of the overflow tail
constexpr int kWcTicket = 10;  // k_stage1 blocks that are done (the last one decides the round)
constexpr int kWcGroup = 11;   // next ray of the round's list for k_stage1
constexpr int kWaveCounters = 12;

constexpr int kQsInt = 5;
constexpr int kSaveStack = 24;

struct QueryArgs {
    const double* origins = nullptr;
    const double* dirs = nullptr;
    long long n = 0;
    int mode = 0;          // BBRT_QUERY_*
    int object = 0;
    int cull = 1;
    void* out = nullptr;   // bbrt_hit[n]
};

}  // namespace bbrt
