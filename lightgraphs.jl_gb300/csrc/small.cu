// small.cu -- Brandes betweenness of graphs whose vertex state fits in one
// SM's shared memory: one thread block per source, no launches per level.
//
// The bit-lane batches of msbfs.cu keep 16 bytes of state per (vertex, source)
// in HBM and pay a 1 KB row gather per contributing edge whatever the number
// of lanes set in it.  Here a block keeps one source's path counts, then its
// dependencies, in shared memory (8 bytes per vertex) and walks every edge
// once per sweep, so the random accesses never leave the SM.  What bounds it
// is instruction issue: 62 % of the issue slots busy with 32 warps per SM
// (ALU pipe 50 %), the rest barriers and fixed latencies; DRAM is idle.
// Measured (exact betweenness, batches -> here): G(10,000, 50,000) 11.7 ->
// 4.10 ms; 24 Barabasi-Albert graphs of up to 20,000 vertices 448 -> 150 ms;
// a 50-vertex digraph 289 -> 36 us.
//
// Replaces, per source, dijkstra_shortest_paths(g, s; allpaths, trackvertices)
// with unit weights (src/shortestpaths/dijkstra.jl:59-141) and
// _accumulate_basic! (src/centrality/betweenness.jl:81-107).  Path counts are
// exact integers and dependencies use the arithmetic of xf64.cuh, as in the
// batches.
//
// Layout.  A plan (built once per graph on the device) relabels the vertices
// by decreasing out-degree and stores 16-bit neighbour ids in groups of four,
// padded with the id n, whose state never takes part: a thread reads four
// neighbours in one 8-byte load, and 32 consecutive vertices of a level have
// rows of about the same length, so a warp can give each thread a vertex (and
// each thread finishes its own vertex) without idling on the longest row.
// The vertices with long rows come first, in plain rows, and are walked by
// whole warps.  The others are cut into chunks of 32 with one row length;
// group j of a chunk's rows is contiguous, so neighbouring vertices' loads
// share sectors, and a row's place follows from one word per chunk, kept in
// shared memory.  Every load of a row is issued before the previous group (or
// vertex) is worked on: with one 1,024-thread block per SM nothing else hides
// the latency of L2.
//
// State of vertex v, two words lo / hi (separate arrays: a 4-byte access uses
// all 32 banks):
//   0                           not reached
//   path count, bits 31 = 0     being counted (the level after the frontier)
//   path count, bit 31          counted; the forward sweep leaves it alone
//   psi, bit 30 = level & 1     finished by the backward sweep
// psi lies in (2^-48, 2^15], so 6 bits of exponent (the low ones of lo) leave
// 56 for the significand: 3 more than binary64 (psi_pack in xf64.cuh).  A vertex of level L has
// successors only at level L + 1, and every other neighbour is a path count
// still or finished with the other parity while level L is swept, so the two
// top bits of hi decide in both sweeps and no level is stored per vertex.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "lgbc_kernels.h"
#include "xf64.cuh"

namespace lgbc {
namespace {

constexpr uint32_t kClosed = 0x80000000u;
constexpr int64_t kSmallColumnBlocks = 8 * 152;
// A count of 2^48 or more ends the attempt: below it no sum over at most
// kSmallMaxN < 2^15 predecessors can reach bit 31 of hi.
constexpr uint32_t kCountLimitHi = 1u << 16;

// ---------------------------------------------------------------------------
// Plan: one block per graph, then all for the columns.
// ---------------------------------------------------------------------------

// One stable pass of a radix sort of n < 2^16 vertex ids by digit(v) in [0, 256),
// by a block of 1,024 threads: warp w takes the w-th of 32 equal stretches of
// `from` (null: the ids in order), counts its digits and then places its ids
// behind those of the warps before it.
constexpr int kPlanWarps = 32;
template <class D>
__device__ __forceinline__ void sort_pass(int n, const int32_t* from, int32_t* to, D digit,
                                          uint16_t (*counts)[256]) {
  __shared__ int digit_base[256];
  constexpr int kAhead = 4;
  const int ln = lane_id(), w = threadIdx.x >> 5;
  const int turns = (n + kPlanWarps * kWarp - 1) / (kPlanWarps * kWarp);
  const int i0 = w * turns * kWarp, i1 = min(n, i0 + turns * kWarp);
  auto walk = [&](auto put) {  // put(id, digit, the lanes of that digit), warp-uniformly
    for (int i = i0; i < i1; i += kAhead * kWarp) {
      int v[kAhead], d[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int at = i + q * kWarp + ln;
        v[q] = at < i1 ? (from ? from[at] : at) : -1;
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) d[q] = v[q] >= 0 ? digit(v[q]) : -1;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        put(v[q], d[q], __match_any_sync(kFull, d[q]));
        __syncwarp();
      }
    }
  };
  for (int k = threadIdx.x; k < kPlanWarps * 256; k += blockDim.x) counts[k >> 8][k & 255] = 0;
  __syncthreads();
  walk([&](int, int d, unsigned peers) {
    if (d >= 0 && ln == __ffs(peers) - 1) counts[w][d] = static_cast<uint16_t>(counts[w][d] + __popc(peers));
  });
  __syncthreads();
  int total = 0;
  if (threadIdx.x < 256)
    for (int k = 0; k < kPlanWarps; ++k) {
      const int c = counts[k][threadIdx.x];
      counts[k][threadIdx.x] = static_cast<uint16_t>(total);
      total += c;
    }
  int incl = total;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (ln >= o) incl += y;
  }
  if (threadIdx.x < 256) digit_base[threadIdx.x] = incl;  // within its 32 digits
  __syncthreads();
  int before = 0;
  if (threadIdx.x < 256)
    for (int k = 0; k < w; ++k) before += digit_base[32 * k + 31];
  __syncthreads();
  if (threadIdx.x < 256) digit_base[threadIdx.x] = before + incl - total;
  __syncthreads();
  walk([&](int v, int d, unsigned peers) {
    const int lead = __ffs(peers) - 1;
    int at = 0;
    if (d >= 0 && ln == lead) {
      at = counts[w][d];
      counts[w][d] = static_cast<uint16_t>(at + __popc(peers));
    }
    at = __shfl_sync(kFull, at, lead);
    if (d >= 0) to[digit_base[d] + at + __popc(peers & ((1u << ln) - 1u))] = v;
  });
  __syncthreads();
}

__global__ void __launch_bounds__(kPlanWarps* kWarp) k_small_plan(const SmallGraph* graphs) {
  extern __shared__ int hist[];  // vertices per row length (in groups), then their first rank
  __shared__ uint16_t counts[kPlanWarps][256];
  __shared__ int total_groups, longest;
  const SmallGraph G = graphs[blockIdx.x];
  const int n = G.n;
  const int bins = (n + 3) / 4 + 1;
  int* first = hist;             // [bins] vertices of the bin
  int* start = hist + bins;      // [bins] first rank of the bin
  int* base = hist + 2 * bins;   // [bins] first group of the bin
  for (int b = threadIdx.x; b < bins; b += blockDim.x) first[b] = 0;
  __syncthreads();
  auto groups_of = [&](int v) { return static_cast<int>((G.rowptr[v + 1] - G.rowptr[v] + 3) >> 2); };
  for (int v = threadIdx.x; v < n; v += blockDim.x) atomicAdd(&first[groups_of(v)], 1);
  __syncthreads();
  // longest rows first: a warp scans the bins downwards
  if (threadIdx.x < kWarp) {
    const int ln = lane_id();
    int rank = 0, grp = 0, most = 0;
    for (int top = bins - 1; top >= 0; top -= kWarp) {
      const int b = top - ln;
      const int c = b >= 0 ? first[b] : 0;
      if (c > 0) most = max(most, b);
      int ic = c, ig = c * b;
#pragma unroll
      for (int o = 1; o < kWarp; o <<= 1) {
        const int yc = __shfl_up_sync(kFull, ic, o), yg = __shfl_up_sync(kFull, ig, o);
        if (ln >= o) {
          ic += yc;
          ig += yg;
        }
      }
      if (b >= 0) {
        start[b] = rank + ic - c;
        base[b] = grp + ig - c * b;
      }
      rank += __shfl_sync(kFull, ic, kWarp - 1);
      grp += __shfl_sync(kFull, ig, kWarp - 1);
    }
    most = static_cast<int>(__reduce_max_sync(kFull, static_cast<unsigned>(most)));
    if (ln == 0) {
      total_groups = grp;
      longest = most;
    }
  }
  __syncthreads();
  // Ranks by id within a length: with ranks as atomics come, the same graph had
  // another plan in every call, and items (ranges of ranks) sums of other sources.
  const int top = longest;
  int32_t* by_low = top < 256 ? G.orig : reinterpret_cast<int32_t*>(G.row);  // rows are written below
  sort_pass(n, nullptr, by_low, [&](int v) { return (top - groups_of(v)) & 255; }, counts);
  if (top >= 256) sort_pass(n, by_low, G.orig, [&](int v) { return (top - groups_of(v)) >> 8; }, counts);
  for (int r = threadIdx.x; r < n; r += blockDim.x) {
    const int v = G.orig[r], b = groups_of(v);
    G.rank[v] = r;
    G.row[r] = static_cast<uint32_t>(base[b] + (r - start[b]) * b);
  }
  if (threadIdx.x == 0) {
    G.row[n] = static_cast<uint32_t>(total_groups);
    *G.nwarp = bins > kSmallWarpGroups + 1 ? start[kSmallWarpGroups] : 0;
  }
  __syncthreads();  // also orders this block's global writes before the reads below
  {
    int live = 0;
    for (int v = threadIdx.x; v < n; v += blockDim.x) live += G.in_rowptr[v + 1] > G.in_rowptr[v] ? 1 : 0;
    live = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(live)));
    if (lane_id() == 0 && live) atomicAdd(G.nlive, live);
  }
  // whole chunks (past n when every row is long)
  const int nw = (*reinterpret_cast<volatile int*>(G.nwarp) + 31) & ~31;
  const int warps = blockDim.x >> 5, ln = lane_id();
  // chunks of the thread-walked vertices: first group and row length (that
  // of the chunk's first vertex, its longest)
  if (threadIdx.x < kWarp) {
    uint32_t at = G.row[min(nw, n)];
    for (int c0 = nw / kWarp; c0 * kWarp < n; c0 += kWarp) {
      const int c = c0 + ln;
      const uint32_t len = c * kWarp < n ? G.row[c * kWarp + 1] - G.row[c * kWarp] : 0u;
      uint32_t incl = len * kWarp;
#pragma unroll
      for (int o = 1; o < kWarp; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (ln >= o) incl += y;
      }
      if (c * kWarp < n) G.chunk[c] = ((at + incl - len * kWarp) << kSmallLenBits) | len;
      at += __shfl_sync(kFull, incl, kWarp - 1);
    }
  }
}

// The columns of the planned rows, a warp per vertex: most of the plan's work.
// One block's plan of 16,384 vertices took 380 us, the two kernels take 72 + 69 on
// cold caches (52 + 69 with ranks as atomics came, 31 + 12 either way for 10,000
// vertices of short rows, which one sort pass orders).
__global__ void __launch_bounds__(256) k_small_columns(const SmallGraph* graphs) {
  const SmallGraph G = graphs[blockIdx.y];
  const int n = G.n;
  const int nw = (*G.nwarp + 31) & ~31, ln = lane_id();
  uint16_t* col = reinterpret_cast<uint16_t*>(G.col);
  for (int v = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5); v < n; v += static_cast<int>(gridDim.x * blockDim.x) >> 5) {
    const int64_t e0 = G.rowptr[v];
    const int deg = static_cast<int>(G.rowptr[v + 1] - e0);
    const int r = G.rank[v];
    int64_t at = G.row[r];
    int len = (deg + 3) >> 2, step = 1;
    if (r >= nw) {
      const uint32_t w = G.chunk[r >> 5];
      at = (w >> kSmallLenBits) + (r & 31);
      len = static_cast<int>(w & ((1u << kSmallLenBits) - 1u));
      step = kWarp;
    }
    for (int i = ln; i < 4 * len; i += kWarp)
      col[4 * (at + static_cast<int64_t>(i >> 2) * step) + (i & 3)] =
          static_cast<uint16_t>(i < deg ? G.rank[G.colidx[e0 + i]] : n);
  }
}

// ---------------------------------------------------------------------------
// Sweeps
// ---------------------------------------------------------------------------

// The shared accesses of a group of four neighbours are written out with
// predicates: as branches around each of the four they cost more instructions
// than the adds themselves.
__device__ __forceinline__ uint32_t lds(uint32_t at) {
  uint32_t x;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(at));
  return x;
}
// *at += add if the sign of h is clear.
__device__ __forceinline__ void red_if_open(uint32_t at, uint32_t add, uint32_t h) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ge.s32 p, %2, 0;\n\t"
      "@p red.shared.add.u32 [%0], %1;\n\t}"
      ::"r"(at), "r"(add), "r"(h) : "memory");
}
// x = *at if h > 0 as a signed number.
__device__ __forceinline__ void lds_if_done(uint32_t& x, uint32_t at, uint32_t h) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.gt.s32 p, %2, 0;\n\t"
      "@p ld.shared.u32 %0, [%1];\n\t}"
      : "+r"(x) : "r"(at), "r"(h));
}
__device__ __forceinline__ uint32_t shared_at(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- Brandes: path counts, then psi, in two words per vertex ---------------
// Reciprocals of the path counts below this come from a table in shared
// memory (most are a handful; the rest are computed).
constexpr int kRecipTable = 512;

struct BrandesState {
  using Sum = PsiSum;         // of psi, while a row is walked
  using Value = xf64;         // the finished sum
  using Early = ulonglong2;   // a vertex's partial sum, loaded ahead of its row
  struct Count {
    uint32_t lo, hi;
  };
  const uint64_t* recip;      // significands of 1 / s, s < kRecipTable
  uint32_t *lo, *hi;
  uint32_t lo_s, hi_s;
  int n;
  ulonglong2* part;
  const double* weight;
  xf64 w;

  static __host__ __device__ size_t words(int64_t n) { return 2 * kRecipTable + 2 * static_cast<size_t>(n + 1); }
  __device__ __forceinline__ BrandesState(uint32_t* sm, const SmallRun& run, const SmallItem& I, const SmallGraph& G)
      : recip(reinterpret_cast<uint64_t*>(sm)), lo(sm + 2 * kRecipTable), hi(lo + G.n + 1), lo_s(shared_at(lo)),
        hi_s(shared_at(hi)), n(G.n), part(run.part + I.part), weight(run.weight), w(xf_zero()) {
    uint64_t* t = reinterpret_cast<uint64_t*>(sm);
    for (int i = threadIdx.x; i < kRecipTable; i += blockDim.x)
      t[i] = xf_recip_u64(static_cast<uint64_t>(i > 0 ? i : 1)).m;
    for (int i = threadIdx.x; i < n; i += blockDim.x) part[i] = make_ulonglong2(0ull, 0ull);
  }
  __device__ __forceinline__ void clear(int si) {
    for (int i = threadIdx.x; i <= 2 * n + 1; i += blockDim.x) lo[i] = 0u;
    if (weight) w = xf_from_bits(static_cast<uint64_t>(__double_as_longlong(weight[si])));
  }
  __device__ __forceinline__ void seed(int s) {
    hi[n] = kClosed;
    lo[s] = 1u;
    hi[s] = kClosed;
  }
  __device__ __forceinline__ Count count(int v) const { return Count{lo[v], hi[v] & ~kClosed}; }

  // A frontier vertex's path count to four neighbours, except those that are
  // closed.  64-bit shared atomics are compare-and-swap loops, so the words
  // are added apart.  With every count of the frontier below 2^16 no sum over
  // fewer than 2^15 predecessors passes 2^31: the adds need no answer and
  // nothing waits for them (NARROW).  Otherwise the low word's old value
  // gives the carry.
  template <bool NARROW> __device__ __forceinline__ void push4(uint2 c, Count f) const {
    // byte offsets of the four state words
    const uint32_t at[4] = {(c.x << 2) & 0x3FFFCu, (c.x >> 14) & 0x3FFFCu, (c.y << 2) & 0x3FFFCu,
                            (c.y >> 14) & 0x3FFFCu};
    uint32_t h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = lds(hi_s + at[k]);
    if (NARROW) {
#pragma unroll
      for (int k = 0; k < 4; ++k) red_if_open(lo_s + at[k], f.lo, h[k]);
      return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t old = 0u;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "setp.ge.s32 p, %3, 0;\n\t"
          "@p atom.shared.add.u32 %0, [%1], %2;\n\t}"
          : "+r"(old) : "r"(lo_s + at[k]), "r"(f.lo), "r"(h[k]) : "memory");
      const uint32_t up = f.hi + (old > ~f.lo ? 1u : 0u);
      if (static_cast<int>(h[k]) >= 0 && up)
        asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(hi_s + at[k]), "r"(up) : "memory");
    }
  }
  // The same for one neighbour (narrow counts); true for its first add.
  __device__ __forceinline__ bool first(uint32_t v, Count f) const {
    return static_cast<int>(hi[v]) >= 0 && atomicAdd(lo + v, f.lo) == 0u;
  }
  __device__ __forceinline__ bool close(int v) const {  // true: the count is 2^16 or more
    hi[v] = kClosed;
    return (lo[v] >> 16) != 0u;
  }
  // Close v if this level counted it; returns whether it did.
  __device__ __forceinline__ bool close_fresh(int v, int* wide, int* stop) const {
    const uint32_t h = hi[v], l = lo[v];
    if (static_cast<int>(h) < 0 || (h | l) == 0u) return false;
    hi[v] = h | kClosed;
    if (h | (l >> 16)) *wide = 1;
    if (h >= kCountLimitHi) *stop = 1;
    return true;
  }

  static __device__ __forceinline__ Sum zero() { return PsiSum{0ull, 0}; }
  // psi of the successors among four neighbours of a vertex of level L into
  // the sum; any other neighbour adds zero.
  __device__ __forceinline__ void pull4(uint2 c, int L, Sum& a) const {
    const uint32_t at[4] = {(c.x << 2) & 0x3FFFCu, (c.x >> 14) & 0x3FFFCu, (c.y << 2) & 0x3FFFCu,
                            (c.y >> 14) & 0x3FFFCu};
    const uint32_t parity = static_cast<uint32_t>((L + 1) & 1) << 30;
    uint32_t h[4], l[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = lds(hi_s + at[k]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      asm volatile(
          "{\n\t.reg .pred p;\n\t.reg .u32 x;\n\t"
          "xor.b32 x, %0, %2;\n\t"
          "setp.lt.u32 p, x, 0x40000000;\n\t"
          "selp.u32 %0, x, 0, p;\n\t"
          "mov.u32 %1, 0;\n\t"
          "@p ld.shared.u32 %1, [%3];\n\t}"
          : "+r"(h[k]), "=&r"(l[k]) : "r"(parity), "r"(lo_s + at[k]));
#pragma unroll
    for (int k = 0; k < 4; ++k) psi_add(a, l[k], h[k], (k & 1) != 0);
  }
  static __device__ __forceinline__ void after32(Sum& a) { psi_norm(a); }
  static __device__ __forceinline__ Value value(Sum a) { return psi_value(a); }
  static __device__ __forceinline__ Value none() { return xf_zero(); }
  static __device__ __forceinline__ Value warp_sum(Value x) { return warp_sum_x(x); }
  __device__ __forceinline__ Early early(int v) const { return part[v]; }
  // psi = 1 / sigma + acc replaces the count; sigma * acc is the dependency.
  __device__ __forceinline__ void finish(int v, int L, Value acc, Early sum) const {
    const uint32_t slo = lo[v], shi = hi[v] & ~kClosed;
    const uint64_t s = (static_cast<uint64_t>(shi) << 32) | slo;
    xf64 r;
    if (shi == 0u && slo < kRecipTable) {
      r.m = recip[slo];
      r.e = 991 + __clz(static_cast<int>(slo)) + (r.m == (1ull << 62) ? 1 : 0);
    } else {
      r = xf_recip_u64(s);
    }
    const xf64 psi = xf_add(acc, r);
    const uint64_t word = psi_pack(psi);
    lo[v] = static_cast<uint32_t>(word);
    hi[v] = static_cast<uint32_t>(word >> 32) | static_cast<uint32_t>(L & 1) << 30;
    if (acc.m == 0) return;
    xf64 d;
    if (shi == 0u) {  // 63 x 32 bits
      const uint64_t p0 = static_cast<uint64_t>(static_cast<uint32_t>(acc.m)) * slo;
      const uint64_t p1 = (acc.m >> 32) * slo + (p0 >> 32);  // below 2^63, at least 2^30
      const int sh = 33 - xf_clz(p1);                        // 0..32
      d.m = (p1 << (32 - sh)) | (static_cast<uint64_t>(static_cast<uint32_t>(p0)) >> sh);
      d.e = acc.e + sh;
    } else {
      d = xf_mul_u64(acc, s);
    }
    if (weight) d = xf_mul(d, w);
    const xf64 t = xf_add(d, xf64{sum.x, static_cast<int32_t>(sum.y)});
    part[v] = make_ulonglong2(t.m, static_cast<unsigned long long>(t.e));
  }
};

// ---- Stress (src/centrality/stress.jl:51-77; the recursion of k_st_delta in
// msbfs.cu): predecessor counts P in 16 bits, bit 15 in the part of bit 31
// above and 1 + (level & 1) once finished, and E = 1 + sum of the successors'
// E in two words, wrapping.  The
// sum times P goes to the result with one 64-bit atomic, whose order cannot
// show.  P < 2^15, as every in-list is shorter.  300 sources on R-MAT 14:
// 2.31 ms as batches, 0.40 ms here.
struct StressState {
  using Sum = unsigned long long;
  using Value = unsigned long long;
  using Early = int;          // the vertex's own id
  struct Count {};
  uint16_t* st;
  uint32_t *lo, *hi;
  uint32_t st_s, lo_s, hi_s;
  int n;
  const int32_t* orig;
  unsigned long long* out;

  static __host__ __device__ size_t words(int64_t n) { return 2 * static_cast<size_t>(n + 1) + static_cast<size_t>(n + 2) / 2; }
  __device__ __forceinline__ StressState(uint32_t* sm, const SmallRun& run, const SmallItem&, const SmallGraph& G)
      : st(reinterpret_cast<uint16_t*>(sm + 2 * (G.n + 1))), lo(sm), hi(sm + G.n + 1), st_s(shared_at(st)),
        lo_s(shared_at(lo)), hi_s(shared_at(hi)), n(G.n), orig(G.orig), out(run.stress) {}
  __device__ __forceinline__ void clear(int) {
    uint32_t* w = reinterpret_cast<uint32_t*>(st);
    for (int i = threadIdx.x; i < (n + 2) / 2; i += blockDim.x) w[i] = 0u;
  }
  __device__ __forceinline__ void seed(int s) {
    st[n] = 0x8000u;
    st[s] = 0x8000u;
  }
  __device__ __forceinline__ Count count(int) const { return Count(); }
  template <bool NARROW> __device__ __forceinline__ void push4(uint2 c, Count) const {
    const uint32_t id[4] = {c.x & 0xFFFFu, c.x >> 16, c.y & 0xFFFFu, c.y >> 16};
    uint32_t h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // the half in the upper 16 bits
      h[k] = lds(st_s + ((id[k] << 1) & ~3u));
      h[k] <<= (~id[k] & 1u) << 4;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) red_if_open(st_s + ((id[k] << 1) & ~3u), (id[k] & 1u) ? 0x10000u : 1u, h[k]);
  }
  __device__ __forceinline__ bool first(uint32_t v, Count) const {
    if (st[v] & 0x8000u) return false;
    const uint32_t sh = (v & 1u) << 4;
    return ((atomicAdd(reinterpret_cast<uint32_t*>(st) + (v >> 1), 1u << sh) >> sh) & 0xFFFFu) == 0u;
  }
  __device__ __forceinline__ bool close(int v) const {
    st[v] |= 0x8000u;
    return false;
  }
  __device__ __forceinline__ bool close_fresh(int v, int*, int*) const {
    const uint16_t p = st[v];
    if (p == 0u || (p & 0x8000u)) return false;
    st[v] = static_cast<uint16_t>(p | 0x8000u);
    return true;
  }
  static __device__ __forceinline__ Sum zero() { return 0ull; }
  __device__ __forceinline__ void pull4(uint2 c, int L, Sum& a) const {
    const uint32_t id[4] = {c.x & 0xFFFFu, c.x >> 16, c.y & 0xFFFFu, c.y >> 16};
    const uint32_t mark = 1u + static_cast<uint32_t>((L + 1) & 1);
    uint32_t h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      h[k] = lds(st_s + ((id[k] << 1) & ~3u));
      h[k] <<= (~id[k] & 1u) << 4;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t done = (h[k] >> 16) == mark ? 1u : 0u;
      uint32_t l = 0u, u = 0u;
      lds_if_done(l, lo_s + 4u * id[k], done);
      lds_if_done(u, hi_s + 4u * id[k], done);
      a += (static_cast<unsigned long long>(u) << 32) | l;
    }
  }
  static __device__ __forceinline__ void after32(Sum&) {}
  static __device__ __forceinline__ Value value(Sum a) { return a; }
  static __device__ __forceinline__ Value none() { return 0ull; }
  static __device__ __forceinline__ Value warp_sum(Value x) { return warp_sum_u64(x); }
  __device__ __forceinline__ Early early(int v) const { return orig[v]; }
  __device__ __forceinline__ void finish(int v, int L, Value acc, Early own) const {
    const unsigned long long e = acc + 1ull;
    lo[v] = static_cast<uint32_t>(e);
    hi[v] = static_cast<uint32_t>(e >> 32);
    const unsigned long long x = acc * (st[v] & 0x7FFFu);
    st[v] = static_cast<uint16_t>(1 + (L & 1));
    if (x) atomicAdd(out + own, x);
  }
};

// One block per item (a range of sources of one graph).  Each source: count
// paths (or predecessors) level by level, then sweep the levels back, adding
// to the item's partial sums (or the result).
template <class S>
__global__ void __launch_bounds__(kSmallMaxThreads, 1) k_small_sweeps(SmallRun run) {
  extern __shared__ uint32_t sm[];
  __shared__ int lvl[2][kSmallMaxLevels + 2];  // level starts: [0] warp-walked vertices, [1] the others
  __shared__ int s_count[kWarp];
  __shared__ int s_item, s_goal, s_own;
  __shared__ int s_stop;                       // 1: the graph was refused or a count is too large, 2: refused here
  __shared__ int s_next[2];                    // [L & 1]: next entry of level L's second list
  __shared__ int s_wide[2];                    // [L & 1]: a count of level L is 2^16 or more
  const int tid = threadIdx.x, T = blockDim.x, ln = lane_id(), wid = tid >> 5, W = T >> 5;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_item = atomicAdd(run.next, 1);
      s_stop = 0;
      if (s_item < run.nitems)  // an earlier source's refusal covers its whole graph
        s_stop = *reinterpret_cast<volatile int*>(run.refused + (run.items ? run.items[s_item].graph : 0));
    }
    __syncthreads();
    if (s_item >= run.nitems) return;
    SmallItem I;
    if (run.items) {
      I = run.items[s_item];
    } else {
      const long long k = run.nsrc;
      I.graph = 0;
      I.begin = static_cast<int>(k * s_item / run.nitems);
      I.end = static_cast<int>(k * (s_item + 1) / run.nitems);
      I.part = static_cast<int64_t>(s_item) * run.graphs[0].n;
    }
    const SmallGraph G = run.graphs[I.graph];
    const int n = G.n;
    S st(sm, run, I, G);
    uint32_t* chunk = sm + S::words(n);
    uint16_t* q = reinterpret_cast<uint16_t*>(chunk + (n + 31) / 32);
    const uint2* const col = G.col;
    // warp-walked ids [0, nw): whole chunks of 32, so that a chunk's
    // discoveries go to one list
    const int nw = (*G.nwarp + 31) & ~31;
    for (int c = nw / kWarp + tid; c * kWarp < n; c += T) chunk[c] = G.chunk[c];
    // the row of a thread-walked vertex: its first group and their number
    auto row_of = [&](uint32_t v, uint32_t& e, int& len) {
      const uint32_t w = chunk[v >> 5];
      e = (w >> kSmallLenBits) + (v & 31u);
      len = static_cast<int>(w & ((1u << kSmallLenBits) - 1u));
    };
    // A warp's next 32 entries of the level's list: the lists are roughly by
    // decreasing row length, so taking them as warps come free evens the
    // warps out.  (i: the lane's entry; its vertex, row and first group.)
    auto fetch = [&](int L, int end, int& i, uint32_t& v, uint32_t& e, int& len, uint2& c) {
      int at = 0;
      if (ln == 0) at = atomicAdd(&s_next[L & 1], kWarp);
      i = __shfl_sync(kFull, at, 0) + ln;
      if (i >= end) return;
      v = q[nw + i];
      row_of(v, e, len);
      if (len > 0) c = col[e];
    };
    // Every count of a level to its successors.
    auto push_level = [&](auto narrow, int L, int a0, int a1, int b1) {
      constexpr bool N = decltype(narrow)::value;
      for (int i = a0 + wid; i < a1; i += W) {
        const int v = q[i];
        const typename S::Count f = st.count(v);
        const uint32_t g1 = G.row[v + 1];
        for (uint32_t e = G.row[v] + ln; e < g1; e += kWarp) st.template push4<N>(col[e], f);
      }
      int i, len = 0;
      uint32_t v = 0, e = 0;
      uint2 c = make_uint2(0u, 0u);
      fetch(L, b1, i, v, e, len, c);
      while (i - ln < b1) {
        const bool on = i < b1;
        const typename S::Count f = st.count(on ? v : n);
        const uint32_t at = e;
        const int groups = on ? len : 0;
        uint2 x = c;
        fetch(L, b1, i, v, e, len, c);
        for (int j = 1; j <= groups; ++j) {
          uint2 nx = x;
          if (j < groups) nx = col[at + 32u * j];
          st.template push4<N>(x, f);
          x = nx;
        }
      }
    };
    for (int si = I.begin; si < I.end && !s_stop; ++si) {
      st.clear(si);
      __syncthreads();
      if (tid == 0) {
        const int s = run.src ? G.rank[run.src[si]] : si;
        st.seed(s);
        const int k = s < nw ? 0 : 1;
        const int own = G.orig[s];
        s_own = own;
        s_goal = *G.nlive + (G.in_rowptr[own + 1] == G.in_rowptr[own] ? 1 : 0);
        q[k ? nw : 0] = static_cast<uint16_t>(s);
        lvl[0][0] = lvl[1][0] = 0;
        lvl[0][1] = 1 - k;
        lvl[1][1] = k;
        s_next[0] = s_wide[0] = s_wide[1] = 0;
      }
      __syncthreads();
      int L = 0;
      for (;;) {
        const int a1 = lvl[0][L + 1], b1 = lvl[1][L + 1];
        // every vertex that any edge enters is reached: nothing is left to find
        if (a1 + b1 == s_goal) break;
        if (tid == 0) s_wide[(L + 1) & 1] = 0;  // last read before the previous barriers
        if (a1 == lvl[0][L] && b1 - lvl[1][L] <= kWarp && !s_wide[L & 1]) {
          // A few short rows: a warp each, and whoever adds to an empty count
          // lists the vertex, which saves the pass over all vertices.
          if (tid < 2) s_count[tid] = 0;
          __syncthreads();
          for (int i = lvl[1][L] + wid; i < b1; i += W) {
            const uint32_t v = q[nw + i];
            const typename S::Count f = st.count(v);
            uint32_t e;
            int len;
            row_of(v, e, len);
            if (ln < len) {
              const uint2 c = col[e + 32u * ln];
              const uint32_t ids[4] = {c.x & 0xFFFFu, c.x >> 16, c.y & 0xFFFFu, c.y >> 16};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const uint32_t w = ids[k];
                if (!st.first(w, f)) continue;
                const int t = w < static_cast<uint32_t>(nw) ? 0 : 1;
                q[(t ? nw + b1 : a1) + atomicAdd(&s_count[t], 1)] = static_cast<uint16_t>(w);
              }
            }
          }
          __syncthreads();
          const int ta = a1 + s_count[0], tb = b1 + s_count[1];
          if (ta == a1 && tb == b1) break;
          auto close = [&](int v) {
            if (st.close(v)) s_wide[(L + 1) & 1] = 1;
          };
          for (int i = a1 + tid; i < ta; i += T) close(q[i]);
          for (int i = b1 + tid; i < tb; i += T) close(q[nw + i]);
          ++L;
          __syncthreads();  // L is even across the block; s_count is read
          if (L + 1 > kSmallMaxLevels) {
            if (tid == 0) s_stop = 2;
            L = 0;
            break;
          }
          if (tid == 0) {
            lvl[0][L + 1] = ta;
            lvl[1][L + 1] = tb;
            s_next[L & 1] = lvl[1][L];
          }
          __syncthreads();
          continue;
        }
        if (s_wide[L & 1])
          push_level(std::false_type(), L, lvl[0][L], a1, b1);
        else
          push_level(std::true_type(), L, lvl[0][L], a1, b1);
        __syncthreads();
        // Close the vertices counted in this level and list them in id order:
        // each warp takes consecutive chunks (32 at most) and keeps chunk j's
        // fresh ids in lane j, the warps' totals give each its place.
        const int nc = (n + kWarp - 1) / kWarp, per = (nc + W - 1) / W;
        const int c0 = wid * per, mine_c = min(per, nc - c0);
        unsigned bits = 0;
        for (int j = 0; j < mine_c; ++j) {
          const int v = (c0 + j) * kWarp + ln;
          const bool fresh = v < n && st.close_fresh(v, &s_wide[(L + 1) & 1], &s_stop);
          const unsigned bal = __ballot_sync(kFull, fresh);
          if (ln == j) bits = bal;
        }
        // counts of both lists in one word: they stay below 2^16
        const int cnt = __popc(bits) << (c0 + ln < nw / kWarp ? 0 : 16);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
          const int y = __shfl_up_sync(kFull, incl, o);
          if (ln >= o) incl += y;
        }
        if (ln == kWarp - 1) s_count[wid] = incl;
        __syncthreads();
        int before = ln < W ? s_count[ln] : 0;
        const int all = before;
        before = ln < wid ? before : 0;
        const int total = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(all)));
        const int place = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(before))) + incl - cnt;
        const int ta = a1 + (total & 0xFFFF), tb = b1 + (total >> 16);
        for (unsigned some = __ballot_sync(kFull, bits != 0u); some; some &= some - 1u) {
          const int j = __ffs(some) - 1;
          const unsigned bal = __shfl_sync(kFull, bits, j);
          const int at = __shfl_sync(kFull, place, j);
          const int id = (c0 + j) * kWarp;
          const int pos = id < nw ? a1 + (at & 0xFFFF) : nw + b1 + (at >> 16);
          if ((bal >> ln) & 1u) q[pos + __popc(bal & ((1u << ln) - 1u))] = static_cast<uint16_t>(id + ln);
        }
        if (ta == a1 && tb == b1) break;
        if (L + 2 > kSmallMaxLevels || s_stop) {
          // the batches take the graph: leave the item
          __syncthreads();  // every thread has read s_stop
          if (tid == 0) s_stop = 2;
          L = 0;
          break;
        }
        ++L;
        if (tid == 0) {
          lvl[0][L + 1] = ta;
          lvl[1][L + 1] = tb;
          s_next[L & 1] = lvl[1][L];
        }
        __syncthreads();
      }
      const int deepest = L;
      for (; L > 0; --L) {
        // for the level after this one (its parity's counter was last used
        // before the previous barrier)
        if (tid == 0) s_next[(L - 1) & 1] = lvl[1][L - 1];
        const int a1 = lvl[0][L + 1], b1 = lvl[1][L + 1];
        int held = 0, mine_v = 0;
        typename S::Value mine = S::none();  // lane j keeps the j-th sum of the warp, to finish 32 at once
        for (int i = lvl[0][L] + wid; i < a1; i += W) {
          const int v = q[i];
          typename S::Value acc = S::none();
          if (L < deepest) {
            typename S::Sum a = S::zero();
            const uint32_t g1 = G.row[v + 1];
            uint32_t e = G.row[v] + ln;
            while (e < g1) {
#pragma unroll 1
              for (int k = 0; k < 8 && e < g1; ++k, e += kWarp) st.pull4(col[e], L, a);
              S::after32(a);
            }
            acc = S::warp_sum(S::value(a));
          }
          if (ln == held) {
            mine = acc;
            mine_v = v;
          }
          if (++held == kWarp) {
            st.finish(mine_v, L, mine, st.early(mine_v));
            held = 0;
          }
        }
        if (ln < held) st.finish(mine_v, L, mine, st.early(mine_v));
        if (L == deepest) {
          for (int i = lvl[1][L] + tid; i < b1; i += T) {
            const int v = q[nw + i];
            st.finish(v, L, S::none(), st.early(v));
          }
        } else {
          int i, len = 0;
          uint32_t v = 0, e = 0;
          uint2 c = make_uint2(0u, 0u);
          fetch(L, b1, i, v, e, len, c);
          while (i - ln < b1) {
            const uint32_t u = v, at = e;
            const bool on = i < b1;
            const int groups = on ? len : 0;
            typename S::Early early{};
            if (on) early = st.early(u);
            uint2 x = c;
            fetch(L, b1, i, v, e, len, c);
            typename S::Sum a = S::zero();
            for (int j = 1; j <= groups; ++j) {
              uint2 nx = x;
              if (j < groups) nx = col[at + 32u * j];
              st.pull4(x, L, a);
              if ((j & 7) == 0) S::after32(a);
              x = nx;
            }
            if (on) st.finish(u, L, S::value(a), early);
          }
        }
        __syncthreads();
      }
      __syncthreads();
    }
    if (tid == 0 && s_stop == 2) {  // refused at the last source begun
      run.refused[I.graph] = 1;
      if (run.deep) run.deep[s_own] = 1;
    }
  }
}

// ---------------------------------------------------------------------------
// Distances from up to 32 sources at once, one bit lane each (or from a source
// set, all in lane 0), of a graph whose three lane words per vertex fit one
// SM's shared memory: a block runs the whole search, pulling each level over
// the in-lists.  Replaces the distance-only batches of msbfs.cu and the
// single BFS of bfs.cu (src/traversals/bfs.jl:95-124) on small graphs, where
// those spend their time on four launches and a host round trip per level.
// A warp takes a chunk of 32 vertices, whose row groups lie side by side, so
// its loads are coalesced without any list of vertices; a chunk that every
// lane has finished is passed over.  Bound: latency of the levels of a few
// blocks (one source), shared-memory loads (many).  Measured against those
// paths: distance sums from all 3,000 vertices of G(3,000, 18,000) 11.6 ms ->
// 82 us, one BFS on G(1,001, 5,003) 222 -> 29 us as a call.
// ---------------------------------------------------------------------------
// ROWS: distances are written (their code costs the statistics 10 % on long rows).
template <bool ROWS>
__global__ void __launch_bounds__(kSmallMaxThreads, 1) k_small_bfs(SmallBfs run) {
  extern __shared__ uint32_t sm[];
  __shared__ unsigned long long s_cnt[kWarp], s_sum[kWarp];
  __shared__ int s_max[kWarp];
  const SmallGraph G = *run.graph;
  const int n = G.n, tid = threadIdx.x, T = blockDim.x, ln = lane_id(), wid = tid >> 5, W = T >> 5;
  uint32_t* vis = sm;
  uint32_t* front = sm + (n + 1);
  uint32_t* next = sm + 2 * (n + 1);
  uint32_t* chunk = sm + 3 * (n + 1);
  const int nc = (n + kWarp - 1) / kWarp;
  const int nw = (*G.nwarp + 31) & ~31;
  const int first = blockIdx.x * kWarp;
  const int nl = run.together ? 1 : min(kWarp, run.nsrc - first);
  const uint32_t full = nl == kWarp ? ~0u : (1u << nl) - 1u;
  const int64_t row0 = static_cast<int64_t>(first) * n;
  int32_t* dist = run.dist ? run.dist + row0 : nullptr;
  long long* dist64 = run.dist64 ? run.dist64 + row0 : nullptr;
  auto put = [&](int64_t at, int32_t d) {
    if (!ROWS) return;
    if (dist) dist[at] = d;
    if (dist64) dist64[at] = d == kUnreached ? INT64_MAX : static_cast<long long>(d);
  };
  for (int i = tid; i < 3 * (n + 1); i += T) sm[i] = 0u;
  for (int c = nw / kWarp + tid; c < nc; c += T) chunk[c] = G.chunk[c];
  if (tid < kWarp) {
    s_cnt[tid] = s_sum[tid] = 0ull;
    s_max[tid] = 0;
  }
  __syncthreads();
  for (int i = tid; i < (run.together ? run.nsrc : nl); i += T) {
    const int own = run.src ? run.src[first + i] : run.few[first + i], r = G.rank[own];
    const uint32_t bit = run.together ? 1u : 1u << i;
    atomicOr(vis + r, bit);
    atomicOr(front + r, bit);
    put(static_cast<int64_t>(run.together ? 0 : i) * n + own, 0);
  }
  __syncthreads();
  // lane b of every warp counts what the warp's vertices add to source b
  unsigned cnt = 0;
  unsigned long long sum = 0;
  int deepest = 0;
  const uint2* const col = G.col;
  for (int level = 1;; ++level) {
    unsigned fresh = 0;  // vertices the level adds to source `ln`
    auto put_level = [&](uint32_t bits, int v) {
      const int own = G.orig[v];
      for (; bits; bits &= bits - 1u) put(static_cast<int64_t>(__ffs(bits) - 1) * n + own, level);
    };
    for (int v = wid; v < min(nw, n); v += W) {
      const uint32_t want = full & ~vis[v];
      uint32_t got = 0;
      if (want) {
        for (uint32_t e = G.row[v] + ln; e < G.row[v + 1]; e += kWarp) {
          const uint2 c = col[e];
          got |= front[c.x & 0xFFFFu] | front[c.x >> 16] | front[c.y & 0xFFFFu] | front[c.y >> 16];
        }
        got = __reduce_or_sync(kFull, got) & want;
      }
      if (ln == 0) {
        next[v] = got;
        if (got) vis[v] |= got;
      }
      fresh += (got >> ln) & 1u;
      if (ROWS && got) {  // lane j: source j's row
        const int own = G.orig[v];
        if ((got >> ln) & 1u) put(static_cast<int64_t>(ln) * n + own, level);
      }
    }
    for (int c = nw / kWarp + wid; c < nc; c += W) {
      const int v = c * kWarp + ln;
      const uint32_t want = v < n ? full & ~vis[v] : 0u;
      uint32_t got = 0;
      if (__any_sync(kFull, want != 0u)) {
        const uint32_t w = chunk[c];
        const int len = static_cast<int>(w & ((1u << kSmallLenBits) - 1u));
        if (v < n) {
          const uint2* row = col + (w >> kSmallLenBits) + ln;
#pragma unroll 4
          for (int j = 0; j < len; ++j) {
            const uint2 x = row[kWarp * j];
            got |= front[x.x & 0xFFFFu] | front[x.x >> 16] | front[x.y & 0xFFFFu] | front[x.y >> 16];
          }
        }
        got &= want;
        if (__any_sync(kFull, got != 0u)) {
          fresh += __popc(warp_transpose32(got));
          if (got) {
            vis[v] |= got;
            if (ROWS) put_level(got, v);
          }
        }
      }
      if (v < n) next[v] = got;
    }
    cnt += fresh;
    sum += static_cast<unsigned long long>(fresh) * static_cast<unsigned>(level);
    if (fresh) deepest = level;
    if (!__syncthreads_or(static_cast<int>(fresh))) break;
    uint32_t* const t = front;
    front = next;
    next = t;
  }
  if (ROWS)
    for (int v = tid; v < n; v += T) {
      const int own = G.orig[v];
      for (uint32_t miss = full & ~vis[v]; miss; miss &= miss - 1u)
        put(static_cast<int64_t>(__ffs(miss) - 1) * n + own, kUnreached);
    }
  if (!run.cnt) return;
  if (cnt) {
    atomicAdd(&s_cnt[ln], static_cast<unsigned long long>(cnt));
    atomicAdd(&s_sum[ln], sum);
    atomicMax(&s_max[ln], deepest);
  }
  __syncthreads();
  if (tid < nl) {
    run.cnt[first + tid] = s_cnt[tid];
    run.dsum[first + tid] = s_sum[tid];
    run.dmax[first + tid] = s_max[tid];
  }
}

// out[orig] = the sum of a graph's partial vectors, in item order.  A block
// takes 32 vertices of graph blockIdx.y; its warps sum interleaved items,
// then warp 0 sums those.
__global__ void __launch_bounds__(256) k_small_sums(const SmallGraph* graphs, const SmallSum* sums,
                                                   const ulonglong2* part, double* out, int* counters,
                                                   int* refused) {
  __shared__ uint64_t sm_m[8][kWarp];
  __shared__ int sm_e[8][kWarp];
  if (counters && blockIdx.x == 0 && threadIdx.x == 0) {
    *refused = counters[1];
    counters[0] = counters[1] = 0;
  }
  const SmallSum S = sums[blockIdx.y];
  const SmallGraph G = graphs[S.graph];
  if (blockIdx.x * kWarp >= G.n) return;
  const int ln = lane_id(), wid = threadIdx.x >> 5;
  const int v = blockIdx.x * kWarp + ln;
  xf64 a = xf_zero();
  if (v < G.n)
    for (int i = wid; i < S.items; i += 8) {
      const ulonglong2 o = part[S.part + static_cast<int64_t>(i) * G.n + v];
      a = xf_add(a, xf64{o.x, static_cast<int32_t>(o.y)});
    }
  sm_m[wid][ln] = a.m;
  sm_e[wid][ln] = a.e;
  __syncthreads();
  if (wid || v >= G.n) return;
  for (int i = 1; i < 8; ++i) a = xf_add(a, xf64{sm_m[i][ln], sm_e[i][ln]});
  double x = __longlong_as_double(static_cast<long long>(xf_to_bits(a)));
  if (S.active >= 0) {
    x += static_cast<double>(S.active);
    if (v < S.active) x += static_cast<double>(G.n) - 2.0;
  }
  out[S.out + G.orig[v]] = x;
}

// CSRs that no handle has validated: one block per graph.
__global__ void __launch_bounds__(256) k_small_check(const SmallGraph* graphs, int* bad) {
  const SmallGraph G = graphs[blockIdx.x];
  const int64_t nnz = G.rowptr[G.n];
  int f = 0;
  for (int v = threadIdx.x; v < G.n; v += blockDim.x) {
    const int64_t d = G.rowptr[v + 1] - G.rowptr[v];
    f |= d < 0 ? 1 : (d > G.n ? 4 : 0);
  }
  for (int64_t e = threadIdx.x; e < nnz; e += blockDim.x)
    f |= G.colidx[e] < 0 || G.colidx[e] >= G.n ? 2 : 0;
  if (f) atomicOr(bad + blockIdx.x, f);
}

}  // namespace

namespace {
// State, chunk words and level lists of an n-vertex graph.
template <class S> size_t sweep_smem(int64_t n) {
  return (S::words(n) + static_cast<size_t>((n + 31) / 32)) * 4 + ((static_cast<size_t>(n) * 2 + 15) & ~size_t(15));
}

template <class S> int sweep_configure(size_t max_dyn_smem) {
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, k_small_sweeps<S>) != cudaSuccess) return 0;
  const size_t room = max_dyn_smem > fa.sharedSizeBytes ? max_dyn_smem - fa.sharedSizeBytes : 0;
  cudaFuncSetAttribute(k_small_sweeps<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room));
  int64_t n = std::min<int64_t>(kSmallMaxN, static_cast<int64_t>(room / 10));
  while (n > 0 && sweep_smem<S>(n) > room) --n;
  return static_cast<int>(n);
}

template <class S> SmallShape sweep_shape(const LaunchCfg& c, int64_t max_n, int64_t items) {
  SmallShape sh{};
  const size_t smem = sweep_smem<S>(max_n);
  // as many warps as the registers allow, split over the blocks that fit and
  // that there are items for
  int64_t blocks = std::min<int64_t>(16, static_cast<int64_t>((227 * 1024) / (smem + 4096)));
  blocks = std::max<int64_t>(1, std::min(blocks, (items + c.sms - 1) / c.sms));
  int threads = static_cast<int>(kSmallMaxThreads / blocks);
  threads = std::max(64, std::min(threads, static_cast<int>((2 * max_n + 31) & ~int64_t(31))));
  threads &= ~31;
  // a warp lists at most 32 chunks of 32 vertices
  const int chunks = static_cast<int>((max_n + kWarp - 1) / kWarp);
  threads = std::max(threads, (chunks + kWarp - 1) / kWarp * kWarp);
  int resident = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_small_sweeps<S>, threads, smem) != cudaSuccess ||
      resident < 1)
    resident = 1;
  sh.threads = threads;
  sh.grid = c.sms * resident;
  return sh;
}

template <class S> int sweep(cudaStream_t s, const SmallShape& sh, const SmallRun& run, int64_t max_n) {
  const int grid = std::min(sh.grid, run.nitems);
  k_small_sweeps<S><<<grid, sh.threads, sweep_smem<S>(max_n), s>>>(run);
  return 1;
}
}  // namespace

// Rows rounded up to groups, and each chunk's rows to its longest: since the
// lengths decrease, that adds at most the first chunk's.
int64_t small_col_groups(int64_t n, int64_t nnz) {
  return (nnz + 3 * n) / 4 + kWarp * (kSmallWarpGroups + 1);
}

size_t small_bfs_smem(int64_t n) {
  return (3 * static_cast<size_t>(n + 1) + static_cast<size_t>((n + 31) / 32)) * 4;
}

int small_bfs_configure(size_t max_dyn_smem) {
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, k_small_bfs<true>) != cudaSuccess) return 0;
  const size_t room = max_dyn_smem > fa.sharedSizeBytes ? max_dyn_smem - fa.sharedSizeBytes : 0;
  cudaFuncSetAttribute(k_small_bfs<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room));
  cudaFuncSetAttribute(k_small_bfs<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room));
  int64_t n = std::min<int64_t>(kSmallMaxN, static_cast<int64_t>(room / 12));
  while (n > 0 && small_bfs_smem(n) > room) --n;
  return static_cast<int>(n);
}

int small_bfs(const LaunchCfg& c, cudaStream_t s, const SmallBfs& run, int64_t n) {
  const int blocks = run.together ? 1 : (run.nsrc + kWarp - 1) / kWarp;
  const size_t smem = small_bfs_smem(n);
  int64_t per_sm = std::min<int64_t>(16, static_cast<int64_t>((227 * 1024) / (smem + 2048)));
  per_sm = std::max<int64_t>(1, std::min<int64_t>(per_sm, (blocks + c.sms - 1) / c.sms));
  int threads = static_cast<int>(kSmallMaxThreads / per_sm);
  threads = std::max(64, std::min(threads, static_cast<int>((n + 31) & ~int64_t(31)))) & ~31;
  (run.dist || run.dist64 ? k_small_bfs<true> : k_small_bfs<false>)<<<blocks, threads, smem, s>>>(run);
  return 1;
}

int small_configure(size_t max_dyn_smem) {
  cudaFuncSetAttribute(k_small_plan, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(max_dyn_smem / 2));
  return sweep_configure<BrandesState>(max_dyn_smem);
}
int small_stress_configure(size_t max_dyn_smem) { return sweep_configure<StressState>(max_dyn_smem); }

int small_plan(cudaStream_t s, const SmallGraph* graphs, int count, int64_t max_n) {
  const size_t bins = static_cast<size_t>((max_n + 3) / 4 + 1);
  k_small_plan<<<count, kPlanWarps * kWarp, 3 * bins * sizeof(int), s>>>(graphs);
  // eight vertices a warp, and no more blocks than are resident
  const int64_t x = std::max<int64_t>(1, std::min((max_n + 63) / 64, kSmallColumnBlocks / count));
  k_small_columns<<<dim3(static_cast<unsigned>(x), static_cast<unsigned>(count)), 256, 0, s>>>(graphs);
  return 2;
}

SmallShape small_shape(const LaunchCfg& c, int64_t max_n, int64_t items) {
  return sweep_shape<BrandesState>(c, max_n, items);
}
int small_brandes(cudaStream_t s, const SmallShape& sh, const SmallRun& run, int64_t max_n) {
  return sweep<BrandesState>(s, sh, run, max_n);
}
SmallShape small_stress_shape(const LaunchCfg& c, int64_t n, int64_t items) {
  return sweep_shape<StressState>(c, n, items);
}
int small_stress(cudaStream_t s, const SmallShape& sh, const SmallRun& run, int64_t n) {
  return sweep<StressState>(s, sh, run, n);
}

int small_check(cudaStream_t s, const SmallGraph* graphs, int count, int* bad) {
  k_small_check<<<count, 256, 0, s>>>(graphs, bad);
  return 1;
}

int small_sums(cudaStream_t s, const SmallGraph* graphs, const SmallSum* sums, int count, int64_t max_n,
               const ulonglong2* part, double* out, int* counters, int* refused) {
  const dim3 grid(static_cast<unsigned>((max_n + kWarp - 1) / kWarp), static_cast<unsigned>(count));
  k_small_sums<<<grid, 256, 0, s>>>(graphs, sums, part, out, counters, refused);
  return 1;
}

}  // namespace lgbc
