// lgbc_kernels.h -- host-side launch wrappers shared by the CUDA translation
// units of the lgbc library.  Every wrapper returns the number of kernels it
// queued, which the API layer counts for lgbc_stats / lgbc_timer_stop.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "lgbc_internal.cuh"

struct lgbc_mlp;

namespace lgbc {

// Path-count representation of a multi-source batch.
enum SigmaKind : int {
  kSigmaNone = 0,    // distances only (gdistances_batch)
  kSigmaU64 = 1,     // exact uint64 path counts, double-float (df32) dependency sums (opt-in)
  kSigmaF64 = 2,     // FP64 path counts and dependencies (replay after overflow)
  kSigmaU64F64 = 3,  // exact uint64 path counts, FP64 dependencies (the default)
};
// The forward sweep only sees the path counts: both uint64 kinds run the same
// forward kernels.
constexpr int fwd_kind(int sk) { return sk == kSigmaU64F64 ? kSigmaU64 : sk; }
// Path counts kept as exact uint64 (an overflow replays the batch in FP64).
constexpr bool u64_counts(int sk) { return sk == kSigmaU64 || sk == kSigmaU64F64; }

// Landmark vertices (highest degree) whose BFS distances order the sources.
constexpr int kLandmarks = 16;

struct LaunchCfg {
  int grid;     // blocks for grid-stride kernels
  int block;    // threads per block
  int sms;      // streaming multiprocessors on the device
};

// ---- multi-source (bit-lane) BFS and Brandes sweeps: msbfs.cu ----------
// Per-batch device buffers.  A batch has 64 * words lanes (words = 1 or 2);
// every lane set is `words` consecutive uint64 (lane l in word l / 64, bit
// l % 64), so the mask of vertex v is at [v * words], and lane l of v's
// path-count / psi row lives at [v * 64 * words + l].  The buffers are sized
// for two words; a one-word batch uses their first half.
struct MsBuffers {
  uint64_t* visit;     // n lane sets: lanes that have reached v
  uint64_t* mb[2];     // n lane sets each: dense level masks, F_L lives in mb[L & 1]
  void* sigma;         // n rows: uint64 or double path counts
  void* psi;           // the rows of sigma: (1 + delta) / sigma takes a count's place
  int32_t* qv;         // cap: concatenated level lists (vertex)
  uint64_t* qm;        // cap lane sets: lanes of that vertex at that level
  unsigned long long* lvl_off;  // n + 3: start of each level's list
  BatchCtl* ctl;       // control block
  const int32_t* lane_src;      // sources of the batch (device)
  unsigned long long cap;       // entries in qv / qm
  const double* lane_w;         // 64 * words lane weights (weighted accumulation) or nullptr
  int64_t lane_w_n;             // > 0: a union of copies of an n-vertex graph, one row of 64
                                // weights per copy (vertex v uses row v / lane_w_n; one word)
  unsigned* claim;              // n, two-word batches: top-down first-discovery flags, kept zero
  int words;                    // 64-bit lane words per vertex: 1 or 2
  int lane_filter;              // 1: bottom-up levels skip lanes absent from the frontier
};

// The active lanes of a batch (word 1 unused in a one-word batch).
struct LaneSet {
  uint64_t w[kMaxWords];
};
// Lanes [0, nl) of a batch with `words` words.
inline LaneSet lane_set(int nl, int words) {
  LaneSet a{};
  for (int j = 0; j < words; ++j) {
    const int k = nl - 64 * j;
    a.w[j] = k >= 64 ? ~0ull : (k <= 0 ? 0ull : ((1ull << k) - 1ull));
  }
  return a;
}

// Vertices with more than hub_degree neighbours ("hubs") are not expanded by
// one warp: their edge lists are cut into kHubChunk-edge work items spread over
// the whole grid, whose partial results are combined with atomics; the last
// item of a hub to finish (a completion counter, no waiting) finalises it.
constexpr int kHubChunk = 256;
struct HubItem {
  int64_t lo, hi;      // edge range [lo, hi) in the CSR the item list belongs to
  int32_t v;           // the hub vertex
  int32_t slot;        // its accumulator slot
  int32_t nitems;      // items of this hub in this list
  int32_t bucket;      // order key (ascending in the list), or 0
};
struct HubData {
  const HubItem* out_items;      // items over out-edges (top-down discovery, dependencies)
  long long n_out;
  const HubItem* in_items;       // items over in-edges (path-count pulls, bottom-up)
  long long n_in;
  unsigned long long* acc;       // slots x 64 * words partial sums (uint64 or FP64 bits), kept zero
  unsigned long long* mask;      // slots x words: OR of discovering lanes, kept zero
  unsigned int* cnt;             // slots: finished items, kept zero
  int hub_degree;                // degree above which a vertex is a hub (INT32_MAX: none)
  int dense_edges;               // chunks with more contributing edges use the transposed gather
  int segmented;                 // 1: low-degree kernels (a warp streams 32 vertices' edges)
};

// sigma_limit: (2^64 - 1) / (max in-degree + 1), the largest path count a
// level may hold without the next level risking 64-bit overflow.
int ms_init(cudaStream_t s, const DevGraph& g, const MsBuffers& b, int nlanes, int sigma_kind,
            unsigned long long sigma_limit, int32_t* dist, int64_t dist_ld);
// Level 0 from explicit (vertex, lane set) seeds (distinct vertices; b.words
// mask words per seed); for disjoint unions of graphs, where one lane holds a
// source in every component.  Distances (dist) only with one word.
int ms_init_seeds(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
                  const int32_t* seed_v, const uint64_t* seed_mask, int64_t nseeds, int sigma_kind,
                  unsigned long long sigma_limit, int32_t* dist, int64_t dist_ld);
// visit[v] = seg_mark[k] (b.words words) for every vertex of segment k
// (vertices [seg_off[k], seg_off[k+1])): the lanes with no source in that
// component.
int ms_premark(const LaunchCfg& c, cudaStream_t s, const MsBuffers& b, const int64_t* seg_off,
               const uint64_t* seg_mark, int64_t nseg);
// Top-down / bottom-up level.  Distances (dist) only with one word.
int ms_topdown(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
               const HubData& hd, const LaneSet& act, int sigma_kind, int32_t* dist,
               int64_t dist_ld);
int ms_bottomup(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
                const HubData& hd, const LaneSet& act, int sigma_kind, int32_t* dist,
                int64_t dist_ld);
int ms_advance(cudaStream_t s, const DevGraph& g, const MsBuffers& b);
// Set ctl->level = maxlevel for the backward sweep (on the device).
int ms_begin_backward(cudaStream_t s, const MsBuffers& b);
// Backward (dependency) step for the level in ctl->level, then level--.
int ms_backward_level(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
                      const HubData& hd, int sigma_kind, double* bc);
// The same without the final level decrement (the body of a device-driven loop).
int ms_backward_body(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
                     const HubData& hd, int sigma_kind, double* bc);

// Device-driven level loops: the control kernels of a CUDA graph whose
// conditional nodes run the forward levels (WHILE `loop` { SWITCH `dir` })
// and the backward levels (WHILE `loop`).
struct LoopParams {
  cudaGraphConditionalHandle loop;  // 1: run another iteration
  cudaGraphConditionalHandle dir;   // forward: 0 top-down, 1 bottom-up, 2 none
  long long n;
  long long nnz;
  double alpha;                     // direction-switch thresholds
  double beta;
  int sigma_kind;
  long long max_levels;             // runaway cap (n + 1)
};
int loop_arm(cudaStream_t s, const MsBuffers& b, const LoopParams& lp);
int loop_advance(cudaStream_t s, const MsBuffers& b, const LoopParams& lp);
int loop_back_arm(cudaStream_t s, const MsBuffers& b, const LoopParams& lp);
int loop_back_advance(cudaStream_t s, const MsBuffers& b, const LoopParams& lp);
// Stress step for the level in ctl->level after a distance-only forward
// sweep (E = 1 + D per (vertex, lane) in the path-count rows), adding the
// stress of level + 1 into `stress` (wrapping uint64); then level--.
int st_backward_level(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const MsBuffers& b,
                      const HubData& hd, unsigned long long* stress);
// After the backward sweep: clear the masks of levels 0 and 1.
int ms_cleanup(const LaunchCfg& c, cudaStream_t s, const MsBuffers& b);
// Per-lane distance statistics of a batch (64 entries each, accumulated):
// vertices reached at levels >= 1, the sum of their levels, the deepest level.
struct LevelStats {
  unsigned long long* cnt;
  unsigned long long* dsum;
  int* dmax;
};
// After a distance-only forward sweep (before ms_cleanup_all).
int ms_level_stats(const LaunchCfg& c, cudaStream_t s, const MsBuffers& b, const LevelStats& st);
// After a distance-only batch: clear visit / masks of every listed vertex.
int ms_cleanup_all(const LaunchCfg& c, cudaStream_t s, const MsBuffers& b);
// After the forward sweep of a one-word batch with path counts (uint64 or
// FP64 kind): sigma_out[l * ld + v] = path count of lane l at v as binary64,
// dist_out[l * ld + v] = its level (dist_out may be null), for every listed
// (vertex, lane); unlisted entries are left as they are.
int ms_export(const LaunchCfg& c, cudaStream_t s, const MsBuffers& b, int sigma_kind,
              double* sigma_out, int32_t* dist_out, int64_t ld);
// Zero visit and both mask buffers outright (after an aborted batch).
int ms_reset_all(cudaStream_t s, const DevGraph& g, const MsBuffers& b);

// ---- Brandes on graphs that fit one SM's shared memory: small.cu ----------
constexpr int kSmallMaxN = 32000;        // 16-bit ids with one to spare; the shared memory bounds n further
constexpr int kSmallMaxThreads = 1024;
constexpr int kSmallMaxLevels = 128;     // levels 0 to 127; a deeper search is left to the batches
constexpr int kSmallWarpGroups = 16;    // rows of more than 4 * this entries are walked by a warp
constexpr int kSmallLenBits = 5;         // holds kSmallWarpGroups
// One SM walks a source's edges alone: at 1.2M entries (20,000 vertices) a
// single source took 529 us against 359 us as a batch, at 0.43M 264 against
// 591 us for 16 sources and 16.3 against 17.0 ms for all 16,384.  (Well below
// the 2^27 groups that a chunk word can place.)
constexpr int64_t kSmallMaxNnz = int64_t(1) << 20;
// A graph and its plan (device pointers): the vertices relabelled by
// decreasing out-degree, their rows in groups of four 16-bit ids.
struct SmallGraph {
  int n;
  const int64_t* rowptr;   // the graph's own out-CSR
  const int32_t* colidx;
  const int64_t* in_rowptr;  // its in-CSR's (rowptr when undirected)
  int32_t* rank;           // n: new id of a vertex
  int32_t* orig;           // n: and back
  uint32_t* row;           // n + 1: first group of a row (warp-walked vertices)
  uint32_t* chunk;         // (n + 31) / 32: first group << kSmallLenBits | row length, per 32 ids
  uint2* col;              // small_col_groups(n, nnz) groups, padded with the id n
  int* nwarp;              // ids below this have rows walked by a warp (zero before the plan)
  int* nlive;              // vertices that some edge enters (likewise)
};
struct SmallItem {
  int graph;               // index of its graph
  int begin, end;          // its sources: positions in SmallRun::src, or ids of the plan
  int64_t part;            // its n partial sums in SmallRun::part (zeroed by the kernel)
};
struct SmallRun {
  const SmallGraph* graphs;
  const SmallItem* items;  // null: nsrc sources of graph 0 in nitems equal parts
  int nitems;
  int nsrc;
  int* next;               // zero: the next item
  int* refused;            // per graph, zero: set when a source is too deep or its counts too large
  uint8_t* deep;           // n, or null: set at such a source (its own id)
  const int32_t* src;      // sources as the graph's own ids, or null
  const double* weight;    // weights of the sources in src, or null
  ulonglong2* part;        // extended-format sums (xf64.cuh): significand, exponent
  unsigned long long* stress;  // stress: n results of graph 0, added to
};
struct SmallShape {
  int grid, threads;
};
// One graph's result: the sum of its items' partial sums, plus the endpoint
// terms of its `active` sources (add_endpoints) when wanted.
struct SmallSum {
  int graph;
  int items;
  int active;              // -1: no endpoint terms; else its first ids in the plan are the sources
  int64_t part;            // items x n
  int64_t out;
};
constexpr int kSmallFew = 8;  // sources that travel with the launch
// Distances on a small graph, 32 sources per block (or one set of sources).
struct SmallBfs {
  const SmallGraph* graph;   // plan of the in-CSR
  const int32_t* src;        // graph's own ids, or null: the first nsrc of few
  int32_t few[kSmallFew];
  int nsrc;
  int together;              // 1: one search from all the sources
  int32_t* dist;             // nsrc (or 1) x n, every entry written; or null
  long long* dist64;         // the same in 64 bits, INT64_MAX where not reached; or null
  unsigned long long* cnt;   // per source: vertices reached at levels >= 1, or null
  unsigned long long* dsum;  //   and the sum
  int* dmax;                 //   and maximum of their levels
};
// The largest n of the kernel on this device (opts it into the shared memory).
int small_bfs_configure(size_t max_dyn_smem);
int small_bfs(const LaunchCfg& c, cudaStream_t s, const SmallBfs& run, int64_t n);
int64_t small_col_groups(int64_t n, int64_t nnz);
// Opt the kernels into the device's shared memory; the largest n they take.
int small_configure(size_t max_dyn_smem);
int small_plan(cudaStream_t s, const SmallGraph* graphs, int count, int64_t max_n);
// Launch shape for `items` items of graphs of up to max_n vertices.
SmallShape small_shape(const LaunchCfg& c, int64_t max_n, int64_t items);
int small_brandes(cudaStream_t s, const SmallShape& sh, const SmallRun& run, int64_t max_n);
// Stress centrality (run.stress) likewise.
int small_stress_configure(size_t max_dyn_smem);
SmallShape small_stress_shape(const LaunchCfg& c, int64_t n, int64_t items);
int small_stress(cudaStream_t s, const SmallShape& sh, const SmallRun& run, int64_t n);
// ORs into bad[i] for graph i: 1 = rowptr decreases, 2 = a column outside
// [0, n), 4 = a row longer than n.
int small_check(cudaStream_t s, const SmallGraph* graphs, int count, int* bad);
// counters, when given, are those of a single-graph run: its refusal goes to
// *refused (which may be pinned host memory, as out may) and both are zeroed
// for the next run.
int small_sums(cudaStream_t s, const SmallGraph* graphs, const SmallSum* sums, int count, int64_t max_n,
               const ulonglong2* part, double* out, int* counters = nullptr, int* refused = nullptr);

// ---- single multi-source BFS (gdistances): bfs.cu ------------------------
// One level per launch (lgbc_gdistances_noalloc).
struct BfsBuffers {
  int32_t* queue;               // n: every level, concatenated
  uint32_t* bm[2];              // (n + 31) / 32 words each: frontier bitmaps
  BatchCtl* ctl;
};
// A whole search in one cooperative launch.
constexpr int kBfsAhead = 4;               // edges a thread has in flight
constexpr int kBfsChunk = 32 * kBfsAhead;  // out-edges a warp takes of a long list
struct BfsSlot {                // one level's frontier, rotating over three
  unsigned long long count, mf, mu;  // vertices, their out-edges and in-edges
  unsigned long long queued;         // those listed in the queue
  unsigned long long big;            // entries << 32 | chunks of the list of long out-lists
};
struct BfsState {               // zeroed before the launch
  GridBarrier barrier;
  BfsSlot slot[3];
  long long td_levels, bu_levels;
};
struct BfsRun {
  int32_t* dist;                // n
  const int32_t* src;
  int64_t nsrc;
  int prefilled;                // 1: the caller filled dist (kUnreached, or another value where
                                // the search must not go); 0: filled here
  int32_t* queue;               // n
  uint32_t* visited;            // the visited bitmap and three level bitmaps of `words` words
  int64_t words;                //   (a multiple of 4, at least (n + 31) / 32)
  int2* big;                    // two lists of big_cap entries: (first chunk, vertex)
  int64_t big_cap;              // at least nnz / kBfsChunk + 1
  BfsState* state;
  double alpha, beta;
  int stage;                    // set by bfs_run: the frontier bitmap fits shared memory
};
// room: bfs_configure's result.
int bfs_run(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, BfsRun r, size_t room);
int bfs_init(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
             const int32_t* src, int64_t nsrc, int32_t* dist);
int bfs_topdown(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
                int32_t* dist);
int bfs_bottomup(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
                 int32_t* dist, int stage_smem);
int bfs_advance(cudaStream_t s, const BfsBuffers& b);
// parents[v] = smallest in-neighbour of v at distance dist[v] - 1 (the
// source: itself; unreached: -1).
int bfs_parents(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const int32_t* dist,
                int32_t* parents);
// p[idx[i]] = value for i < count.
int scatter_i32(const LaunchCfg& c, cudaStream_t s, int32_t* p, const int32_t* idx, int64_t count,
                int32_t value);
// Opt the kernels into the device's shared memory; the bytes k_bfs_run may stage.
size_t bfs_configure(size_t max_dyn_smem);

// Set the thread-local message returned by lgbc_last_error() (api.cu).
void set_last_error(const char* msg);

// ---- small utilities: util.cu ----------------------------------------------
// ORs into *bad: 1 = rowptr decreases somewhere, 2 = a column index is not in
// [0, n), 4 = rowptr[0] != 0 or rowptr[n] != nnz.
int validate_csr(const LaunchCfg& c, cudaStream_t s, const int64_t* rowptr, const int32_t* colidx,
                 int64_t n, int64_t nnz, int* bad);
// out[i] = in[i] in 64 bits, INT64_MAX where in[i] is kUnreached (16-byte aligned arrays).
int widen_dist(const LaunchCfg& c, cudaStream_t s, const int32_t* in, int64_t count, int64_t* out);
int fill_i32(const LaunchCfg& c, cudaStream_t s, int32_t* p, int64_t count, int32_t value);
// The CSR of a disjoint union of `copies` copies of an n-vertex graph (copy
// r = vertices [r n, (r + 1) n)): rp1[copies n + 1], c1[copies nnz]; n > 0.
int replicate_csr(const LaunchCfg& c, cudaStream_t s, const int64_t* rp0, const int32_t* c0,
                  int64_t n, int64_t nnz, int64_t copies, int64_t* rp1, int32_t* c1);
// The hub items of such a union from those of one graph with n vertices, nnz
// entries and nslots hubs: bucket by bucket and copy by copy in each, as the
// union's own list is ordered, or copy by copy.
int replicate_items(const LaunchCfg& c, cudaStream_t s, const HubItem* in, int64_t count, int64_t copies, int64_t n,
                    int64_t nnz, int64_t nslots, bool buckets, HubItem* out);
// out[v] = sum over r < copies of stacked[r * n + v] (a fixed order).
int sum_copies(const LaunchCfg& c, cudaStream_t s, const double* stacked, int64_t n, int64_t copies,
               double* out);
// out[r * nl + j] = dist[j * ld + src[r]] for r < k, j < nl.
int gather_cols(const LaunchCfg& c, cudaStream_t s, const int32_t* dist, int64_t ld, int nl,
                const int32_t* src, int64_t k, int32_t* out);
int fill_f64(const LaunchCfg& c, cudaStream_t s, double* p, int64_t count, double value);
// bc[v] += k_act for every v, then bc[s] += n - 2 for each active source s:
// the endpoint terms of _accumulate_endpoints! summed over the sources.
int add_endpoints(const LaunchCfg& c, cudaStream_t s, double* bc, int64_t n,
                  const int32_t* active_src, int64_t k_act);
// The same for a disjoint union of graphs: segment i = vertices [seg_off[i],
// seg_off[i+1]) gets seg_add[i] (its active-source count) everywhere, and each
// active source src[j] gets src_add[j] (its graph's n - 2) more.
int add_endpoints_many(const LaunchCfg& c, cudaStream_t s, double* bc, const int64_t* seg_off,
                       const double* seg_add, int64_t nseg, const int32_t* src,
                       const double* src_add, int64_t nsrc);

// ---- learned source proposal: learned.cu ----------------------------------
// deg[v] = neighbours other than v; *loops |= 1 if v has a self-loop.
int core_degree(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, int32_t* deg, int* loops);
// Core numbers from the degrees in core (h-index passes until none is
// lowered), in one cooperative launch.
constexpr int kCoreCached = 256;       // vertices with more neighbour entries are hubs
struct CoreSlot {                      // one pass, rotating over three
  unsigned long long small, hubs;      // vertices to search
  unsigned long long log, hub_log;     // vertices lowered
};
struct CoreState {                     // zeroed before the launch
  GridBarrier barrier;
  CoreSlot slot[3];
  unsigned long long all_hubs;         // entries of CoreRun::all_hubs
  long long passes;
  int loops;                           // a vertex has a self-loop (core_degree)
};
struct CoreRun {
  int32_t* core;                       // n
  uint32_t* flag;                      // (n + 31) / 32 words
  int32_t* small[2];                   // n each
  int32_t* hubs[2];                    // hub_cap each
  int32_t* all_hubs;                   // hub_cap
  int32_t *log_v, *log_old;            // n
  int32_t *hub_v, *hub_old;            // hub_cap
  CoreState* state;
  long long max_passes;                // more means a fault
};
// At most this many vertices have more than kCoreCached entries.
inline int64_t core_hub_cap(int64_t nnz, int directed) { return (directed ? 2 * nnz : nnz) / kCoreCached + 1; }
int core_run(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const CoreRun& r);
// terms: n float2 of scratch; all_hubs / state: as core_run left them.
int features(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const CoreRun& r, float2* terms,
             float4* feat);

// MLP parameter layout (floats): W1[64][4], b1[64], W2[64][64], b2[64], W3[64], b3.
constexpr int kMlpHidden = 64;
constexpr int kMlpW1 = 0;
constexpr int kMlpB1 = kMlpW1 + kMlpHidden * 4;
constexpr int kMlpW2 = kMlpB1 + kMlpHidden;
constexpr int kMlpB2 = kMlpW2 + kMlpHidden * kMlpHidden;
constexpr int kMlpW3 = kMlpB2 + kMlpHidden;
constexpr int kMlpB3 = kMlpW3 + kMlpHidden;
constexpr int kMlpParams = kMlpB3 + 1;                  // 4545
constexpr int kMlpParamsPadded = (kMlpParams + 3) & ~3;
constexpr int kGradRows = kMlpHidden;                   // rows per gradient block
constexpr int kGradThreads = 2 * kMlpHidden;            // two threads per row
static_assert(kMlpParams == 4545, "parameter count");

struct MlpNorm {
  float mu[4];
  float isd[4];   // 1 / stdev
};
struct AdamStep {
  float lr, beta1, beta2, eps;
  float bc1, bc2;  // bias corrections 1 - beta^t
};
int mlp_forward(const LaunchCfg& c, cudaStream_t s, const float4* x, int64_t rows,
                const __nv_bfloat16* P, const MlpNorm& nm, float* y);
// Opt the gradient kernel into its dynamic shared memory (once per device).
int mlp_configure();
// One step on rows [r0, r0 + B): residuals e, their mean (center, one
// float), block partials part, the loss, the reduced gradient (grad may be
// null) and, when master is not null, an Adam update of master / Pw / m1 / m2.
int mlp_train_step(cudaStream_t s, const float4* x, const float* target, int64_t r0, int B,
                   const __nv_bfloat16* P, const MlpNorm& nm, float* e, float* center,
                   float* part, float* loss, float* grad, float* master, __nv_bfloat16* Pw,
                   float* m1, float* m2, const AdamStep& st);
int mlp_to_bf16(cudaStream_t s, const float* master, __nv_bfloat16* P);
// Weights and standardisation of an MLP handle (mlp.cu), for graph calls.
struct MlpView {
  const __nv_bfloat16* P;
  MlpNorm norm;
  int device;
};
int mlp_view(const lgbc_mlp* m, MlpView* out);

// Proposal scratch: tiles of the scan; fscratch needs tiles + 1 floats, tsum
// tiles doubles, scal 1 double.
int64_t proposal_tiles(int64_t n);
int proposal_build(cudaStream_t s, const float* y, int64_t n, double eps, float* fscratch,
                   double* e, double* tsum, double* scal, double* p, double* cdf);
// systematic: draw i uses u_i = (i + U) / k with one uniform U, else k
// independent uniforms.
int proposal_sample(cudaStream_t s, const double* cdf, const double* p, int64_t n, int64_t k,
                    uint64_t seed, bool systematic, int32_t* src, double* w);

// ---- graph ingest on the device: ingest.cu -------------------------------------
// Bit width B of the vertex ids in the 64-bit arc keys (u << B) | v.
int ingest_bits(int64_t n);
// 8-byte words of scratch for the calls below on at most `count` keys.
int64_t ingest_scratch_words(int64_t count);
// Arc keys of an edge list (2 per edge for an undirected graph; a self-loop
// keeps one); *bad |= 1 for ids outside [0, n).
int ingest_make_keys(const LaunchCfg& c, cudaStream_t s, const int32_t* src, const int32_t* dst,
                     int64_t m, int64_t n, int B, int directed, unsigned long long* keys, int* bad);
int ingest_swap_keys(const LaunchCfg& c, cudaStream_t s, const unsigned long long* in, int64_t count,
                     int B, unsigned long long* out);
// Stable LSD radix sort by bits [bit0, bits); keys / alt are swapped as passes
// run (on return `keys` holds the sorted keys).
int radix_sort(cudaStream_t s, unsigned long long*& keys, unsigned long long*& alt, int64_t count,
               int bit0, int bits, int64_t* scratch);
// *nkept = distinct keys (no sentinel) of a sorted list; scratch is for ingest_emit.
int ingest_count(cudaStream_t s, const unsigned long long* keys, int64_t count, int64_t* scratch, int64_t* nkept);
// The distinct keys, and their low halves as columns.
int ingest_emit(cudaStream_t s, const unsigned long long* keys, int64_t count, const int64_t* scratch, int B,
                int32_t* colidx, unsigned long long* kept);
// The low halves of all keys.
int ingest_columns(const LaunchCfg& c, cudaStream_t s, const unsigned long long* keys, int64_t count, int B,
                   int32_t* colidx);
// rowptr[0..n] of sorted distinct keys.
int ingest_rows(const LaunchCfg& c, cudaStream_t s, const unsigned long long* keys, int64_t count, int64_t n,
                int B, int64_t* rowptr);

}  // namespace lgbc
