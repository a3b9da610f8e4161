// api_internal.h -- shared internals of the C ABI translation units
// (api.cu, api_many.cu, api_learned.cu, api_more.cu): error reporting,
// device allocation, per-handle workspaces, the graph handle itself, and the
// host-side helpers of the level loops that several entry points share.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <utility>
#include <vector>


#include "lgbc.h"
#include "lgbc_kernels.h"

namespace lgbc::api {

using namespace lgbc;

inline thread_local std::string g_last_error;

inline int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

inline int cuda_fail(cudaError_t e, const char* what) {
  return fail(LGBC_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define LGBC_CUDA(call)                                   \
  do {                                                    \
    cudaError_t _e = (call);                              \
    if (_e != cudaSuccess) return cuda_fail(_e, #call);   \
  } while (0)

#define LGBC_TRY(expr)          \
  do {                          \
    int _rc = (expr);           \
    if (_rc != LGBC_OK) return _rc; \
  } while (0)

template <class T>
int dev_alloc(T** p, size_t count) {
  *p = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), count * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return fail(LGBC_ENOMEM, std::string("cudaMalloc of ") + std::to_string(count * sizeof(T)) +
                                 " bytes failed: " + cudaGetErrorString(e));
  }
  return LGBC_OK;
}

template <class T>
void dev_free(T*& p) {
  if (p) cudaFree(p);
  p = nullptr;
}

// Host passes over the vertices of a large graph run on several threads:
// f(part, begin, end) for `parts` contiguous chunks of [0, n), part 0 on the
// calling thread.  Returns the number of parts (1 below 2^16 elements).
template <class F>
int parallel_parts(int64_t n, F&& f) {
  const unsigned hw = std::thread::hardware_concurrency();
  const int parts = n < (int64_t(1) << 16) ? 1 : static_cast<int>(std::max(1u, std::min(8u, hw)));
  std::vector<std::thread> pool;
  for (int p = 1; p < parts; ++p)
    pool.emplace_back([&, p] { f(p, n * p / parts, n * (p + 1) / parts); });
  f(0, int64_t(0), n / parts);
  for (auto& t : pool) t.join();
  return parts;
}

// Multi-source workspace (msbfs.cu): lane sets sized for two words per
// vertex / list entry; path-count / psi rows for `sigma_words` words.
struct MsWorkspace {
  uint64_t* visit = nullptr;
  uint64_t* mb0 = nullptr;
  uint64_t* mb1 = nullptr;
  void* sigma = nullptr;
  int32_t* qv = nullptr;
  uint64_t* qm = nullptr;
  unsigned long long* lvl_off = nullptr;
  BatchCtl* ctl = nullptr;
  unsigned* claim = nullptr;    // two-word batches only
  unsigned long long cap = 0;
  int sigma_words = 0;          // 0: no path-count rows yet

  void release() {
    dev_free(visit);
    dev_free(mb0);
    dev_free(mb1);
    if (sigma) cudaFree(sigma);
    sigma = nullptr;
    dev_free(qv);
    dev_free(qm);
    dev_free(lvl_off);
    dev_free(ctl);
    dev_free(claim);
    cap = 0;
    sigma_words = 0;
  }
};

// Hub work items (see HubItem in lgbc_kernels.h) and their accumulators.
struct HubTable {
  HubItem* out_items = nullptr;
  int64_t n_out = 0;
  HubItem* in_items = nullptr;   // == out_items for undirected graphs
  int64_t n_in = 0;
  unsigned long long* acc = nullptr;  // one allocation with mask and cnt
  unsigned long long* mask = nullptr;
  unsigned int* cnt = nullptr;
  int64_t nslots = 0;
  int built_for = -1;            // hub_degree the table was built with
  int built_order = -1;          // and hub_order
  void release() {
    if (in_items && in_items != out_items) cudaFree(in_items);
    dev_free(out_items);
    in_items = nullptr;
    dev_free(acc);
    mask = nullptr;
    cnt = nullptr;
    n_out = n_in = nslots = 0;
    built_for = -1;
    built_order = -1;
  }
};

struct BfsWorkspace {
  int32_t* queue = nullptr;
  uint32_t* bits = nullptr;     // the visited bitmap and the three level bitmaps
  int2* big = nullptr;          // the two lists of long out-lists
  BfsState* state = nullptr;
  void release() {
    dev_free(queue);
    dev_free(bits);
    dev_free(big);
    dev_free(state);
  }
};

// Learned-proposal state of a graph (learned.cu): core numbers, features,
// scores, the proposal p and its CDF, and scan scratch.
struct LearnedWorkspace {
  CoreRun run{};                           // core numbers and the lists of their passes
  float4* feat = nullptr;
  float* y = nullptr;
  float* fscr = nullptr;
  double* e = nullptr;
  double* tsum = nullptr;
  double* scal = nullptr;
  double* p = nullptr;
  double* cdf = nullptr;
  int32_t* samp = nullptr;
  double* samp_w = nullptr;
  int64_t samp_cap = 0;
  bool built = false;
  int64_t core_passes = 0;
  void release() {
    dev_free(run.core);
    dev_free(run.flag);
    for (int i = 0; i < 2; ++i) {
      dev_free(run.small[i]);
      dev_free(run.hubs[i]);
    }
    dev_free(run.all_hubs);
    dev_free(run.log_v);
    dev_free(run.log_old);
    dev_free(run.hub_v);
    dev_free(run.hub_old);
    dev_free(run.state);
    dev_free(feat);
    dev_free(y);
    dev_free(fscr);
    dev_free(e);
    dev_free(tsum);
    dev_free(scal);
    dev_free(p);
    dev_free(cdf);
    dev_free(samp);
    dev_free(samp_w);
    samp_cap = 0;
    built = false;
  }
};

// The relabelled rows of a small graph's out-CSR or in-CSR (small.cu).
struct SmallPlan {
  SmallGraph view{};                // host copy of *graph
  SmallGraph* graph = nullptr;
  int* counters = nullptr;          // [0] warp-walked ids, [1] live vertices
  void release() {
    dev_free(view.rank);
    dev_free(view.orig);
    dev_free(view.row);
    dev_free(view.chunk);
    dev_free(view.col);
    dev_free(graph);
    dev_free(counters);
  }
};

// Sources that a per-source kernel has refused (too deep, or counts too large):
// a call that has one runs as batches, without another attempt.  Where most
// sources are refused, all calls do.
struct DeepSources {
  std::vector<uint8_t> known;       // empty: none yet
  int64_t count = 0, taken = 0;     // refused sources; sources of the calls taken
  bool given_up() const { return count >= 32 && 16 * count > taken; }
  bool among(const std::vector<int32_t>& src) const {
    if (count == 0) return false;
    for (int32_t v : src)
      if (known[static_cast<size_t>(v)]) return true;
    return false;
  }
};

// Plans and workspace of the shared-memory kernels for small graphs.
struct SmallWorkspace {
  SmallPlan out, in;                // in: digraphs only
  SmallSum* sum = nullptr;
  int64_t items = 0;                // parts of a call that *sum was written for
  // [0] next item, [1] refused (zero between calls); [2, 3] for stress; then
  // the refused sources of both, n bytes each (zero at first)
  int* counters = nullptr;
  ulonglong2* part = nullptr;       // partial sums, one n-vector per item
  int64_t part_cap = 0;
  DeepSources deep, stress_deep;
  void release() {
    out.release();
    in.release();
    dev_free(sum);
    items = 0;
    dev_free(counters);
    dev_free(part);
    part_cap = 0;
  }
};

// A device-driven level loop instantiated for one configuration.
struct LoopKey {
  int backward;                 // 0 forward sweep, 1 backward (dependency) sweep
  int sigma_kind;
  LaneSet act;
  const int32_t* dist;
  int64_t dist_ld;
  const double* bc;
  MsBuffers b;                  // lane_src and lane_w zeroed: not used inside the loop
  HubData hd;
  double alpha, beta;
};
struct LoopGraph {
  LoopKey key;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int td_kernels = 0;           // kernels per top-down / bottom-up / backward level
  int bu_kernels = 0;
  int body_kernels = 0;
  uint64_t last_use = 0;
  void release() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
  }
};

}  // namespace lgbc::api

namespace lgbc::api {
// Explicit (vertex, lane mask) seeds on the device, for unions of graphs;
// the vertices are distinct (a vertex that starts several lanes has them all
// in its mask).
struct Seeds {
  const int32_t* v = nullptr;
  const uint64_t* mask = nullptr;   // one lane set per seed (1 or 2 words: the batch's)
  int64_t count = 0;
  // optional premark of seedless lanes per component (unions of graphs)
  const int64_t* seg_off = nullptr;
  const uint64_t* seg_mark = nullptr;  // one lane set per component
  int64_t nseg = 0;
  // stacked unions with lane weights: one row of 64 * words weights per copy
  // of an lane_w_n-vertex graph, lane_w_count weights in all
  int64_t lane_w_n = 0;
  int64_t lane_w_count = 0;
};
// Forward-sweep export of a one-word batch with path counts (lgbc_path_counts):
// the batch stops after its forward sweep, with sigma / dist written per lane.
struct PathExport {
  double* sigma = nullptr;
  int32_t* dist = nullptr;  // may be null
  int64_t ld = 0;           // row length (n)
};
}  // namespace lgbc::api

namespace lgbc::api {
constexpr size_t kPinnedCtl = 4096;      // room for the control block mirror
constexpr size_t kPinnedOut = size_t(1) << 16;
constexpr int64_t kPinnedSources = 4096;
static_assert(sizeof(BatchCtl) + 16 <= kPinnedCtl, "pinned layout");
constexpr lgbc_tuning kDefaultTuning{14.0, 24.0, 256, 128, 32, 0, 1, 1, 1 << 21, 2, 0};
}

struct lgbc_graph {
  int device = 0;
  int64_t n = 0;
  int64_t nnz = 0;
  int directed = 0;
  cudaStream_t stream = nullptr;
  int64_t* d_rowptr = nullptr;
  int32_t* d_colidx = nullptr;
  int64_t* d_in_rowptr = nullptr;   // == d_rowptr for undirected graphs
  int32_t* d_in_colidx = nullptr;
  std::vector<uint8_t> has_degree;  // degree(g, v) > 0, host copy for filtering
  std::mutex mu;
  lgbc::api::MsWorkspace ms;
  lgbc::api::BfsWorkspace bfs;
  lgbc::api::HubTable hubs;
  lgbc::api::LearnedWorkspace learned;
  lgbc::api::SmallWorkspace small;
  int64_t small_max_n = 0;          // largest graph of the per-source kernel on this device
  int64_t small_stress_max_n = 0, small_bfs_max_n = 0;  // and of the stress and distance kernels
  int64_t max_out = 0, max_in = 0;  // largest out- and in-list
  int64_t long_in = 0;              // in-lists that the shared-memory kernels walk by warps
  int64_t linked = 0;               // vertices of degree > 0
  int32_t* d_src = nullptr;         // device copy of a call's source list
  int64_t d_src_cap = 0;
  double* d_bc = nullptr;           // device result buffer for host-buffer calls
  int32_t* d_dist = nullptr;        // device distance buffer (gdistances)
  int64_t d_dist_cap = 0;
  int64_t* d_wide = nullptr;        // the same in 64 bits
  int64_t d_wide_cap = 0;
  unsigned long long* d_stats = nullptr;  // distance statistics of a call's sources
  int64_t d_stats_cap = 0;
  // pinned host memory, one allocation: the mirror of a control block, then
  // what small calls exchange with their kernels without a copy
  lgbc::BatchCtl* h_ctl = nullptr;
  unsigned char* h_out = nullptr;         // kPinnedOut bytes of results
  int32_t* h_src = nullptr;               // kPinnedSources source ids
  cudaEvent_t ev_start = nullptr, ev_stop = nullptr;
  int64_t launches = 0;             // running count of kernels launched
  int64_t launches_at_start = 0;
  lgbc::LaunchCfg cfg{};
  size_t max_smem = 0;
  size_t bfs_room = 0;              // shared memory the BFS may stage its bitmap in
  unsigned long long sigma_limit = ~0ull;  // (2^64 - 1) / (max in-degree + 1)
  lgbc_stats stats{};
  lgbc_tuning tune = lgbc::api::kDefaultTuning;
  lgbc_graph* stack = nullptr;        // R copies of this graph (stacked batches)
  int64_t stack_copies = 0;
  std::vector<int32_t> h_active;      // the last call's ordered active sources
  std::vector<double> h_weights;      // their weights (weighted calls; empty otherwise)
  double* d_lw_fixed = nullptr;       // lane weights of the running batch (cached graphs)
  int64_t d_lw_cap = 0;
  cudaStream_t cap_stream = nullptr;  // stream used to capture level-loop graphs
  std::vector<lgbc::api::LoopGraph> loops;       // cached device-driven level loops
  uint64_t loop_clock = 0;
  std::vector<int32_t> landmarks;   // the highest-degree vertices (source ordering)
  int32_t* d_lmdist = nullptr;      // landmarks x n BFS distances, computed on first use

  lgbc::DevGraph dev() const {
    return lgbc::DevGraph{n, nnz, d_rowptr, d_colidx, d_in_rowptr, d_in_colidx};
  }
};

namespace lgbc::api {

// Helpers shared by the entry points (api.cu).
int check_graph(const lgbc_graph* g);
int use_device(lgbc_graph* g);
int check_sources(const lgbc_graph* g, const int32_t* src, int64_t nsrc);
int ensure_src(lgbc_graph* g, int64_t count);
// Multi-source workspace; with need_sigma, path-count / psi rows for batches
// of up to 64 * words lanes.
int ensure_ms(lgbc_graph* g, bool need_sigma, int words = 1);
int ensure_bfs(lgbc_graph* g);
int ensure_dist(lgbc_graph* g, int64_t count);
int ensure_hubs(lgbc_graph* g);
HubData hub_data(const lgbc_graph* g);
int read_ctl(lgbc_graph* g, const BatchCtl* dctl);
int check_launch(lgbc_graph* g);
MsBuffers ms_buffers(lgbc_graph* g, const int32_t* lane_src, const double* lane_w = nullptr);
// One multi-source batch: forward level loop, then (with sigma) the backward
// dependency sweep into bc.  Returns LGBC_OK, or 1 when the batch must be
// replayed with FP64 path counts.  lane_w (sigma batches): per-lane weights of
// the accumulation into bc; stats (distance-only batches): per-lane distance
// statistics, accumulated; stress (distance-only batches): the stress sweep;
// pexp (one-word batches with path counts): export the forward sweep and
// skip the dependency sweep.
int run_ms_batch(lgbc_graph* g, const int32_t* lane_src, int nl, int sigma_kind, double* bc,
                 int32_t* dist, int64_t dist_ld, const Seeds& seeds = Seeds(),
                 const double* lane_w = nullptr, const LevelStats* stats = nullptr,
                 unsigned long long* stress = nullptr, const PathExport* pexp = nullptr);
// The path-count / dependency kind of a Brandes batch on this handle: exact
// uint64 path counts with FP64 dependencies (default) or, with the
// dependency_df32 tuning field, double-float dependencies.
inline int dep_kind(const lgbc_graph* g) {
  return g->tune.dependency_df32 ? kSigmaU64 : kSigmaU64F64;
}
// Brandes over the active sources already on the device (g->d_src[0, k)),
// accumulating into bc_dev (zeroed here); with d_w, source i's dependencies
// are scaled by d_w[i].
int run_betweenness(lgbc_graph* g, int64_t k_act, int endpoints, double* bc_dev,
                    const double* d_w = nullptr);
// Brandes over g->h_active (with g->h_weights unless empty), in the order that
// suits the path taken, into bc_dev; host_out, when given, receives the result
// (bc_dev is then scratch) and the call is blocking.
int accumulate_active(lgbc_graph* g, int endpoints, double* bc_dev, double* host_out);
// Validate and keep the sources of degree > 0 (betweenness.jl:58) in g->h_active.
int filter_sources(lgbc_graph* g, const int32_t* src, int64_t nsrc);
// Order g->h_active (and g->h_weights) for batches and copy the sources to g->d_src.
int order_sources(lgbc_graph* g);
void reset_stats(lgbc_graph* g);
void finish_stats(lgbc_graph* g);
int init_handle(lgbc_graph* g, int64_t n, int directed);
// Host rowptr copies are required; colidx copies may be null (copied back
// from the device when the hub items need them).
int finish_handle(lgbc_graph* g, const int64_t* rowptr, const int64_t* in_rowptr,
                  const int32_t* colidx = nullptr, const int32_t* in_colidx = nullptr);
// Whether the shared-memory distance kernel takes nsrc searches (rows: whose
// distances are wanted one by one), and the call (run: everything but the graph).
bool small_bfs_applies(const lgbc_graph* g, int64_t nsrc, bool rows);
int run_small_bfs(lgbc_graph* g, SmallBfs run);
// Whether the per-source kernel takes Brandes calls of this handle, and such a
// call: the k sources at src (device or pinned memory) into out (likewise); it
// waits for the stream and returns 1 when it refuses.
bool same_tuning(const lgbc_tuning& a, const lgbc_tuning& b);
bool small_applies(const lgbc_graph* g);
int run_small(lgbc_graph* g, const int32_t* src, int64_t k, double* out, const double* d_w);
// Stress over g->h_active into d_stress (zeroed by the caller) by the
// per-source kernel: 1 when it does not take the graph (d_stress zero again).
int run_small_stress(lgbc_graph* g, unsigned long long* d_stress);
int upload_sources(lgbc_graph* g);
// A call's source list to g->d_src; the next one waits until the stream has it.
int copy_sources(lgbc_graph* g, const int32_t* src, int64_t k);
// Level-synchronous BFS over dg from g->d_src[0, nsrc) into g->d_dist.
// prefilled: the caller has filled it (kUnreached, and any other value on
// vertices the search must treat as already visited).  finish_bfs waits for
// the stream and checks the search.
int run_bfs(lgbc_graph* g, const DevGraph& dg, int64_t nsrc, bool prefilled = false);
int finish_bfs(lgbc_graph* g);
int prepare_bfs(lgbc_graph* g, const int32_t* src, int64_t nsrc);

}  // namespace lgbc::api
