// Internal declarations shared by the mesh_to_sdf_b200 CUDA sources.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cmath>
#include <memory>
#include <string>
#include <vector>

#include "../../include/m2s.h"
#include "m2s_geo.cuh"
#include "m2s_reach.cuh"

namespace m2s {

// Kernels OR (1u << status) into a device word; the host maps the lowest set
// bit back to a status code.
__host__ __device__ constexpr uint32_t bit(int status) { return 1u << status; }

// One triangle, 48 bytes, read with three 128-bit loads.
//   a.w : degenerate kind (TRI_*), as int bits
//   b.w : triangle index in the crate's triangle order, as uint bits
//   c.w : unused (0)
struct __align__(16) TriRec {
  float4 a, b, c;
};

// Internal LBVH node, 64 bytes: both child boxes live in the parent so one
// node fetch tests both children.  l_lo.w / l_hi.w hold the left / right
// child references (uint bits); LEAF_BIT marks a leaf (index into the
// LBVH-ordered triangle array).  r_lo.w / r_hi.w hold the squared distances up
// to which the left / right child's pillbox may prune (0: never).
struct __align__(16) BvhNode {
  float4 l_lo, l_hi, r_lo, r_hi;
};
constexpr uint32_t LEAF_BIT = 0x80000000u;

// A second bound of a node's children, 32 bytes each (left, then right): a
// pillbox that holds the child's triangles, centre c, unit axis n, half height
// h and radius r.  An axis-aligned box is loose by about a triangle's size, so
// for a point far from the mesh every leaf within that much of the nearest
// distance is visited; a patch of a surface is flat, and its pillbox is loose
// by the patch's sagitta only.  Searches prune by both bounds (pill_dist2 in
// m2s_query.cu).
//   a : c.xyz | h and r rounded up to 16 bits each (h high), slack included
//   b : n.xyz | squared distance up to which the bound may prune (0: never; also in the node)
struct __align__(16) Pill {
  float4 a, b;
};
// Children of more leaves than this have no pillbox (a large patch is not
// flat, and building it would read every leaf once per level).
constexpr uint32_t kPillLeaves = 256;
// A pillbox prunes a search whose best distance is at most the least reach of
// its triangles (m2s_reach.cuh), where the reference's own f32 distance is
// proven to lie above the bound.  The box test before it puts the query within
// that distance of the child's box, so a box of at most kReachSpan reaches keeps
// every triangle of the child within the distances the proof covers.
// Slack of a pillbox per unit of coordinate magnitude: the node's share is in
// h and r, the query's is added by the search.
constexpr float kPillSlack = 0x1p-17f;
// A pillbox is used when its half height is below this share of the box's.
constexpr float kPillFlat = 0.5f;

// Device view of a resident mesh.
struct MeshView {
  const TriRec* tris;    // crate triangle order
  const TriRec* stris;   // LBVH leaf order
  const BvhNode* nodes;  // n_tris - 1 internal nodes (node 0 is the root)
  const Pill* pills;     // two per internal node, or NULL (the nodes' limits are then 0)
  uint32_t n_tris;
  uint32_t root;  // 0, or LEAF_BIT | 0 for a single triangle
};

// Thread-local error detail for m2s_last_error().
void set_error(const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define M2S_CUDA(call)                                    \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return ::m2s::cuda_fail(e_, #call); \
  } while (0)

// Stream-ordered device allocation from the library's memory pool.
int dev_alloc(void** p, size_t bytes, cudaStream_t s);
void dev_free(void* p, cudaStream_t s);

template <class T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  cudaStream_t s = nullptr;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n), s(o.s) { o.p = nullptr; }
  DevBuf& operator=(DevBuf&& o) noexcept {
    release();
    p = o.p, n = o.n, s = o.s;
    o.p = nullptr;
    return *this;
  }
  int alloc(size_t count, cudaStream_t st) {
    release();
    s = st;
    n = count;
    if (count == 0) return M2S_OK;
    return dev_alloc((void**)&p, count * sizeof(T), st);
  }
  void release() {
    if (p) dev_free(p, s);
    p = nullptr;
    n = 0;
  }
  ~DevBuf() { release(); }
};

// ---- LBVH build (m2s_lbvh.cu) ----------------------------------------------

struct MeshInput {
  const float* d_vertices;  // device, 3 * n_vertices
  uint64_t n_vertices;
  const void* d_indices;  // device or NULL
  int index_bits;         // 0 / 16 / 32
  int topology;           // 0 list / 1 strip
  uint64_t n_tris;
};

struct DeviceMesh {
  DevBuf<TriRec> tris, stris;
  DevBuf<BvhNode> nodes;
  DevBuf<Pill> pills;  // none where memory did not suffice or the server gave them back
  uint32_t n_tris = 0;
  uint32_t root = 0;
  MeshView view() const { return {tris.p, stris.p, nodes.p, pills.p, n_tris, root}; }
};

// Gives the pillboxes of a mesh that no search reads back; searches then prune
// by the boxes alone, with the same results.  Waits for the stream.
int drop_pills(DeviceMesh* m, cudaStream_t s);

// Builds the triangle records and the LBVH.  d_status receives status bits.
// with_tree = false builds the triangle records only (grid path, brute force).
int build_device_mesh(const MeshInput& in, DeviceMesh* out, uint32_t* d_status, cudaStream_t s,
                      bool with_tree = true, bool with_pills = true);

// ---- sorting (m2s_sort.cu) ----------------------------------------------------

// Stable LSD radix sort of (key, value) pairs over the low key_bits bits.
// keep_keys = false leaves the keys in no order (the values alone are wanted).
int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint64_t n, int key_bits, cudaStream_t s, bool keep_keys = true);

// The same with another limit of the look-back's polls (0: every count from the
// keys) and, with big, the 64-bit tile words of 2^30 pairs and more (tests).
int radix_sort_pairs_with(uint32_t* keys, uint32_t* vals, uint64_t n, int key_bits, uint32_t max_polls, bool big,
                          cudaStream_t s);

// order: 0 .. n - 1 stably by f32::total_cmp of d; minmax (2 floats, may be
// NULL): the extremes of the values that are no NaN.
int sort_floats(const float* d, uint64_t n, uint32_t* order, float* minmax, cudaStream_t s);

// ---- point queries (m2s_query.cu) -------------------------------------------

// budget >= 0 overrides the process-wide node budget (g_query_budget) for
// this call only: the autotuner times candidates without publishing them.
int query_points(const MeshView& m, int accel, int sign, const float* d_q, uint64_t nq, float* d_out,
                 float* d_vec, uint8_t* d_inside, uint32_t* d_status, cudaStream_t s, int64_t budget = -1);

// Node visits a query may spend in the one-thread-per-query pass before it is
// continued one warp per query (0 disables the second pass).
extern std::atomic<uint32_t> g_query_budget;
// The budget a batch of nq queries uses: `base` from 2^20 queries up,
// base * sqrt(nq / 2^20) from 2^18 and base * nq / 2^19 below, at least
// min(24, base) (0 stays 0: no warp pass).  A batch whose queries all have a thread from the
// start waits for its longest searches, which the warp pass finishes sooner;
// the more queries, the more the thread pass's throughput counts (budgets 24 /
// 64 / 128 / 192: star s6, RtreeBvh, 20,000 queries 0.35 / 0.39 / 0.43 / 0.45
// ms, 100,000 0.88 / 0.75 / 0.58 / 0.61; the terrain strip, Rtree, 20,000
// 0.31 / 0.39 / 0.50 / 0.61 ms, 130,000 1.41 / 1.37 / 1.28 / 1.23; star s6,
// Bvh(Normal), 100,000 1.50 / 1.15 / 0.67 / 0.71).
inline uint32_t effective_query_budget(uint32_t base, uint64_t nq) {
  if (base == 0) return 0;
  const double f = nq >= (1ull << 20)   ? 1.0
                   : nq >= (1ull << 18) ? std::sqrt((double)nq / (double)(1ull << 20))
                                        : (double)nq / (double)(1ull << 19);
  return std::max((uint32_t)(base * f + 0.5), std::min<uint32_t>(24, base));
}
// Node budgets the query autotuner tries.
constexpr int kQueryBudgetCandidates = 8;
constexpr uint32_t kQueryBudgets[kQueryBudgetCandidates] = {0, 64, 256, 512, 1024, 1536, 2048, 4096};
// Profiling (m2s_set_profiling, per host thread): whether it is on, and the
// traversal counts of the last point query made with it on:
// [queries, search node fetches, search triangle tests, sign node fetches,
// sign triangle tests].
bool profiling_enabled();
// [queries, the four traversal counts, the seven FP64-audit counts]
void record_query_stats(const uint64_t stats[12]);

// allow_alloc = false takes no scratch buffer: d_out then holds what chunks merge.
int brute_force_sdf(const MeshView& m, int sign, const float* d_q, uint64_t nq, float* d_out,
                    uint32_t* d_status, cudaStream_t s, bool allow_alloc = true);

// ---- grid (m2s_grid.cu) ------------------------------------------------------

struct GridDesc {
  float first[3];
  float size[3];
  uint64_t n[3];
  // Cell count, saturated at UINT64_MAX when the product overflows.
  uint64_t cells() const {
    unsigned __int128 c = (unsigned __int128)n[0] * n[1];
    if (c > UINT64_MAX) return UINT64_MAX;
    c *= n[2];
    return c > UINT64_MAX ? UINT64_MAX : (uint64_t)c;
  }
};

// stats: [seed updates, relax rounds, states relaxed, neighbour proposals,
// ray hits, overflow restarts, kernel launches, far-list redistributions,
// rounds relaxed by one block alone, largest list relaxed in one round,
// proposals dropped because the neighbour holds the proposing triangle,
// proposals dropped by the distance bound, then the FP64 audit's seven
// counters (zero unless GridTuning::fp64_audit): ray tests, ambiguous ray
// tests, ray tests FP64 decides otherwise, cells whose Raycast vote the FP64
// decisions flip, cells whose Voronoi region was audited, ambiguous region
// choices, region choices FP64 makes otherwise].  phase_ms (may be NULL)
// receives device time of [seeding, propagation, rays, finalize].
constexpr int kGridStats = 19;
int grid_sdf(const MeshView& m, const GridDesc& g, int sign, float* d_out, uint32_t* d_status, cudaStream_t s,
             uint64_t stats[kGridStats], float phase_ms[4]);

// Knobs that change speed, never results.
struct GridTuning {
  int blocks_per_sm = 0;             // cooperative blocks per SM (0: occupancy limit)
  uint32_t cells_per_block = 1024;   // cooperative grid = ceil(cells / this) blocks, at least one per SM
  uint32_t list_capacity = 0;        // entries per bucket list (0: derived from the cell count)
  // A batch runs as jobs ("waves") of at most this many cells each (a larger
  // grid alone), which bounds a job's keys (8 bytes per cell) and lists.
  uint64_t wave_cells = 1ull << 27;
  // Relax rounds of at most this many states run on one block, with block
  // barriers only (0: every round on every block).
  uint32_t solo_max = 64;
  // Drop proposals that a per-triangle distance bound proves cannot win
  // before their closest-point evaluation, in the filtered kernel variant
  // (off: the plain variant; results are identical either way).
  bool bound_filter = false;
  // Audit every ray test and every cell's Voronoi region against an f32
  // error bound and re-decide the ambiguous ones in FP64 (counts only; the
  // output does not change).
  bool fp64_audit = false;
};

struct GridRunInfo {
  bool overflow = false;
  uint64_t seeds = 0, rounds = 0, entries = 0, evals = 0, ray_hits = 0, far_phases = 0, launches = 0, solo_rounds = 0,
           max_list = 0, log_n = 0, filter_same = 0, filter_bound = 0;
  uint64_t audit[7] = {0, 0, 0, 0, 0, 0, 0};
};

// A set of (mesh, grid) pairs computed together: one cell index space (grid k
// starts at the sum of the cells of grids 0..k-1, which is also where its
// output starts in d_out) and one triangle array.  prepare() allocates and
// uploads everything; enqueue() queues the whole pipeline on a stream with no
// host synchronisation, so it can be captured into a CUDA graph; read_state()
// waits for the stream and reports whether the bucket lists overflowed, in
// which case the caller raises the capacity and runs enqueue() again (the
// rerun starts from scratch, so results never depend on the capacity).
class GridJob {
 public:
  GridJob();
  ~GridJob();
  GridJob(const GridJob&) = delete;
  GridJob& operator=(const GridJob&) = delete;
  // out_offsets[k] (NULL: back to back from 0) is where grid k's values start in d_out.
  int prepare(const MeshView* meshes, uint32_t n, const GridDesc* grids, int sign, float* d_out, uint32_t* d_status,
              cudaStream_t s, const GridTuning& tune, const uint64_t* out_offsets = nullptr);
  int alloc_lists(cudaStream_t s);
  int enqueue(cudaStream_t s, cudaEvent_t* ev5);
  int read_state(cudaStream_t s, GridRunInfo* info);
  uint32_t capacity() const;
  void set_capacity(uint32_t cap);
  uint64_t cells() const;
  uint64_t device_bytes() const;  // workspace held by the job (lists included)
  unsigned cooperative_blocks() const;
  unsigned max_cooperative_blocks() const;
  void set_cooperative_blocks(unsigned blocks);  // clamped to [1, max_cooperative_blocks()]
  int sign() const;
  uint32_t grids() const;
  uint32_t threads() const;  // of a propagation block
  // Profiling: record every propagation step (kind and size, and the time it
  // was chosen) in a device log of `cap` steps.
  int enable_round_log(uint32_t cap, cudaStream_t s);
  int read_round_log(std::vector<uint32_t>* out, uint32_t n, cudaStream_t s);

 private:
  struct Impl;
  Impl* p;
};

// Runs a job to completion (restarting with larger lists on overflow).
int run_grid_job(GridJob& job, cudaStream_t s, uint64_t stats[kGridStats], float phase_ms[4]);

// Waves of a batch: grid indices per job, largest grids first, first fit into
// jobs of at most wave_cells cells (a larger grid alone).
std::vector<std::vector<uint32_t>> plan_waves(const GridDesc* grids, uint32_t n, uint64_t wave_cells);

// One prepared job per wave of a batch (outputs back to back in d_out, in the
// order of `grids`).
int prepare_waves(const MeshView* meshes, uint32_t n, const GridDesc* grids, int sign, float* d_out,
                  uint32_t* d_status, cudaStream_t s, const GridTuning& tune,
                  std::vector<std::unique_ptr<GridJob>>* jobs);

// n (mesh, grid) pairs, wave by wave; results back to back in d_out.
int grid_sdf_batch(const MeshView* meshes, uint32_t n, const GridDesc* grids, int sign, float* d_out,
                   uint32_t* d_status, cudaStream_t s, uint64_t stats[kGridStats], float phase_ms[4],
                   const GridTuning& tune);

// Validates a grid description for the device path (32-bit cell indices).
int check_grid(const GridDesc& g);

// Blocks of the propagation kernel that fit on one SM (its occupancy limit).
int propagate_blocks_per_sm(int sign);

// Entries per bucket list of a job of `cells` cells (before any overflow
// restart), and the device bytes of such a job's workspace.
uint32_t default_list_capacity(uint64_t cells);
uint64_t grid_job_bytes(uint64_t cells);

// Process-wide grid knobs (m2s_set_grid_tuning), read as a copy under a lock:
// a caller may change them while other threads (the server's) run grids.
GridTuning grid_tuning();
void set_grid_tuning(const GridTuning& t);

// ---- host API helpers (m2s_api.cu) -------------------------------------------

// M2S_OK when the current device is compute capability 10.x.
int require_device();
// Records the counters / phase times of the last grid call of this thread.
void record_grid_stats(const uint64_t stats[kGridStats]);
float* grid_phase_slot();  // NULL unless profiling is on
void record_round_log(const std::vector<uint32_t>& log);
int status_from_bits(uint32_t bits);

}  // namespace m2s

// Resident mesh behind the m2s_mesh handle.
struct m2s_mesh {
  int device = 0;
  int accel = 0;
  int sign = 0;
  m2s::DeviceMesh mesh;
};

namespace m2s {

}  // namespace m2s
