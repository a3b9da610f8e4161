// ingest.cu -- graph ingest on the device: a CSR built from an edge list.
//
// Replaces the host-side flattening of add_edge!-built adjacency lists for
// large graphs: SimpleGraph / SimpleDiGraph keep every neighbour list sorted
// and free of duplicates (src/SimpleGraphs/simplegraph.jl:445-461,
// simpledigraph.jl:414-429), and an undirected self-loop is stored once.
// Every arc becomes a 64-bit key (u << B) | v with B = bit width of n; the keys
// are sorted by an LSD radix sort (8-bit digits, stable tile scatter), equal
// keys collapse in one scan that writes the columns, and the row starts are
// found by bisection in what is left.  The in-CSR of a digraph needs half the
// digits: the arcs are in order of u already, so a stable sort by v suffices.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lgbc_kernels.h"

namespace lgbc {
namespace {

constexpr int kRsThreads = 256;
constexpr int kRsItems = 16;                       // keys per thread per tile, at most
constexpr int kRsWarps = kRsThreads / 32;
constexpr unsigned long long kSentinel = ~0ull;    // "no arc" (sorts last)

// ---- arcs --------------------------------------------------------------------
// Undirected: slot 2i = (u, v), slot 2i + 1 = (v, u), or the sentinel for a
// self-loop (stored once).  Directed: slot i = (u, v).  *bad |= 1 when an id
// is outside [0, n).
__global__ void k_make_keys(const int32_t* src, const int32_t* dst, int64_t m, int64_t n, int B,
                            int directed, unsigned long long* keys, int* bad) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < m;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t u = src[i], v = dst[i];
    const bool ok = u >= 0 && u < n && v >= 0 && v < n;
    if (!ok) atomicOr(bad, 1);
    const unsigned long long uu = ok ? static_cast<unsigned long long>(u) : 0ull;
    const unsigned long long vv = ok ? static_cast<unsigned long long>(v) : 0ull;
    if (directed) {
      keys[i] = ok ? ((uu << B) | vv) : kSentinel;
    } else {
      keys[2 * i] = ok ? ((uu << B) | vv) : kSentinel;
      keys[2 * i + 1] = (ok && u != v) ? ((vv << B) | uu) : kSentinel;
    }
  }
}

// Swap the two halves of every key: (u, v) -> (v, u) (the in-CSR of a digraph).
__global__ void k_swap_keys(const unsigned long long* in, int64_t count, int B,
                            unsigned long long* out) {
  const unsigned long long mask = (1ull << B) - 1ull;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const unsigned long long k = in[i];
    out[i] = ((k & mask) << B) | (k >> B);
  }
}

// ---- LSD radix sort, one 8-bit digit per pass ------------------------------
// hist[d * tiles + t] = keys of tile t with digit d.
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const unsigned long long* keys, int64_t count,
                                                        int shift, int items, int64_t tiles,
                                                        uint32_t* hist) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * items * kRsThreads;
  for (int r = 0; r < items; ++r) {
    const int64_t i = base + r * kRsThreads + threadIdx.x;
    if (i < count) atomicAdd(&h[(keys[i] >> shift) & 255ull], 1u);
  }
  __syncthreads();
  hist[static_cast<int64_t>(threadIdx.x) * tiles + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter: tile t writes its digit-d keys from off[d * tiles + t] on,
// in tile order.  The tile is walked in rounds of 256 keys (one per thread,
// in thread order); within a round a key's rank is the keys of the same
// digit in earlier warps plus its rank among its warp's peers.
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const unsigned long long* keys,
                                                           int64_t count, int shift, int items,
                                                           int64_t tiles,
                                                           const int64_t* off,
                                                           unsigned long long* out) {
  __shared__ int64_t run[256];                 // next slot of each digit for this tile
  __shared__ uint32_t wc[kRsWarps][256];       // per-warp digit counts of the round
  const int t = threadIdx.x, ln = t & 31, wp = t >> 5;
  run[t] = off[static_cast<int64_t>(t) * tiles + blockIdx.x];
  for (int w = 0; w < kRsWarps; ++w) wc[w][t] = 0u;
  __syncthreads();
  const int64_t base = static_cast<int64_t>(blockIdx.x) * items * kRsThreads;
  for (int r = 0; r < items; ++r) {
    const int64_t i = base + r * kRsThreads + t;
    const bool ok = i < count;
    const unsigned long long k = ok ? keys[i] : 0ull;
    const int d = ok ? static_cast<int>((k >> shift) & 255ull) : 256;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int rank = __popc(peers & ((1u << ln) - 1u));
    if (ok && rank == 0) wc[wp][d] = static_cast<uint32_t>(__popc(peers));
    __syncthreads();
    if (ok) {
      int64_t pos = run[d] + rank;
      for (int w = 0; w < wp; ++w) pos += wc[w][d];
      out[pos] = k;
    }
    __syncthreads();
    uint32_t tot = 0;
    for (int w = 0; w < kRsWarps; ++w) {
      tot += wc[w][t];
      wc[w][t] = 0u;
    }
    run[t] += tot;
    __syncthreads();
  }
}

// ---- scans ---------------------------------------------------------------------
constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanTileN = kScanThreads * kScanPer;

__device__ __forceinline__ int64_t block_exclusive(int64_t v, int64_t* red, int64_t* total) {
  const int ln = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (ln >= o) x += y;
  }
  if (ln == 31) red[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int64_t s = red[ln];
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (ln >= o) s += y;
    }
    red[ln] = s;
  }
  __syncthreads();
  const int64_t incl = x + (wid > 0 ? red[wid - 1] : 0);
  *total = red[31];
  __syncthreads();
  return incl - v;
}

// What is scanned: the cells of a histogram, or 1 for the first copy of each
// key (sentinels dropped).
struct Cells {
  const uint32_t* in;
  __device__ __forceinline__ int64_t operator()(int64_t i) const { return in[i]; }
};
struct FirstCopies {
  const unsigned long long* keys;
  __device__ __forceinline__ int64_t operator()(int64_t i) const {
    const unsigned long long k = keys[i];
    return k != kSentinel && (i == 0 || keys[i - 1] != k) ? 1 : 0;
  }
};

// Exclusive scan, phase 1: tile sums.
template <class In>
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(In in, int64_t count, int64_t* sums) {
  __shared__ int64_t red[32];
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTileN +
                       static_cast<int64_t>(threadIdx.x) * kScanPer;
  int64_t s = 0;
  for (int q = 0; q < kScanPer; ++q)
    if (base + q < count) s += in(base + q);
  int64_t total;
  block_exclusive(s, red, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Phase 2 (one block): exclusive scan of the tile sums in place; *grand = total.
__global__ void __launch_bounds__(kScanThreads) k_scan_sums_excl(int64_t* sums, int64_t tiles,
                                                                 int64_t* grand) {
  __shared__ int64_t red[32];
  int64_t carry = 0;
  for (int64_t b0 = 0; b0 < tiles; b0 += kScanThreads) {
    const int64_t i = b0 + threadIdx.x;
    const int64_t v = i < tiles ? sums[i] : 0;
    int64_t total;
    const int64_t ex = block_exclusive(v, red, &total);
    if (i < tiles) sums[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0 && grand) *grand = carry;
}

// Phase 3: put(i, in at i, its exclusive prefix).
struct StorePrefix {
  int64_t* out;
  __device__ __forceinline__ void operator()(int64_t i, int64_t, int64_t run) const { out[i] = run; }
};
// The kept arcs: columns, and the keys without gaps.
struct EmitArc {
  const unsigned long long* keys;
  unsigned long long mask;  // of the low half of a key
  int32_t* colidx;
  unsigned long long* kept;
  __device__ __forceinline__ void operator()(int64_t i, int64_t is_first, int64_t run) const {
    if (!is_first) return;
    const unsigned long long k = keys[i];
    colidx[run] = static_cast<int32_t>(k & mask);
    kept[run] = k;
  }
};
template <class In, class Put>
__global__ void __launch_bounds__(kScanThreads) k_scan_out(In in, int64_t count, const int64_t* sums, Put put) {
  __shared__ int64_t red[32];
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTileN +
                       static_cast<int64_t>(threadIdx.x) * kScanPer;
  int64_t loc[kScanPer];
  int64_t s = 0;
  for (int q = 0; q < kScanPer; ++q) {
    loc[q] = base + q < count ? in(base + q) : 0;
    s += loc[q];
  }
  int64_t total;
  int64_t run = sums[blockIdx.x] + block_exclusive(s, red, &total);
  for (int q = 0; q < kScanPer; ++q)
    if (base + q < count) {
      put(base + q, loc[q], run);
      run += loc[q];
    }
}

// The whole scan of a short histogram by one block, up to kShortPer cells a
// thread (count is a multiple of 256).
constexpr int kShortPer = 16;
__global__ void __launch_bounds__(kScanThreads) k_scan_short(const uint32_t* in, int count, int64_t* out) {
  __shared__ int64_t red[32];
  const int per = ((count + kScanThreads - 1) / kScanThreads + 3) & ~3;  // whole uint4
  const int base = static_cast<int>(threadIdx.x) * per;
  uint4 c[kShortPer / 4];
  int64_t s = 0;
#pragma unroll
  for (int q = 0; q < kShortPer / 4; ++q) {
    c[q] = make_uint4(0u, 0u, 0u, 0u);
    if (4 * q < per && base + 4 * q < count) c[q] = reinterpret_cast<const uint4*>(in + base)[q];
    s += static_cast<int64_t>(c[q].x) + c[q].y + c[q].z + c[q].w;
  }
  int64_t total;
  int64_t run = block_exclusive(s, red, &total);
#pragma unroll
  for (int q = 0; q < kShortPer / 4; ++q)
    if (4 * q < per && base + 4 * q < count) {
      int64_t* o = out + base + 4 * q;
      o[0] = run;
      o[1] = run += c[q].x;
      o[2] = run += c[q].y;
      o[3] = run += c[q].z;
      run += c[q].w;
    }
}

// ---- rows ------------------------------------------------------------------------
// rowptr[v] = sorted keys below (v, 0), for v in [0, n]: neighbouring threads
// bisect along the same path, so the keys they read are in the caches.
__global__ void k_rows(const unsigned long long* keys, int64_t count, int64_t n, int B, int64_t* rowptr) {
  for (int64_t v = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; v <= n;
       v += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const unsigned long long key = static_cast<unsigned long long>(v) << B;
    int64_t lo = 0, len = v < n ? count : 0;
    while (len > 0) {
      const int64_t half = len >> 1;
      const bool below = keys[lo + half] < key;
      lo = below ? lo + half + 1 : lo;
      len = below ? len - half - 1 : half;
    }
    rowptr[v] = v < n ? lo : count;
  }
}

__global__ void k_columns(const unsigned long long* keys, int64_t count, int B, int32_t* colidx) {
  const unsigned long long mask = (1ull << B) - 1ull;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    colidx[i] = static_cast<int32_t>(keys[i] & mask);
}

}  // namespace

// ---- host side ----------------------------------------------------------------------
int ingest_bits(int64_t n) {
  int B = 1;
  while ((1ll << B) <= n) ++B;  // ids < n <= 2^B - 1, so no key equals the sentinel
  return B;
}

static int64_t scan_tiles(int64_t count) { return (count + kScanTileN - 1) / kScanTileN; }

// Keys per thread of a sort tile: a long list keeps a tile's 256 cells cheap
// against its keys, a short one spreads over up to 64 blocks (50,000 keys: 13 us
// a scatter in 12 full tiles, 3.3 us in 49).
static int rs_items(int64_t count) {
  return static_cast<int>(std::min<int64_t>(kRsItems, std::max<int64_t>(1, (count + 64 * kRsThreads - 1) / (64 * kRsThreads))));
}
static int64_t rs_tiles(int64_t count) {
  const int64_t tile = static_cast<int64_t>(rs_items(count)) * kRsThreads;
  return (count + tile - 1) / tile;
}
// What one block scans at once: a launch in place of three.
constexpr int64_t kScanShort = kScanThreads * kShortPer;

// Words of 8 bytes: the offsets, the cells (half as many) and the tile sums.
// Fewer keys can make more tiles, but then 64 at most.
int64_t ingest_scratch_words(int64_t count) {
  const int64_t cells = 256 * std::max<int64_t>(64, rs_tiles(count));
  return cells + cells / 2 + std::max(scan_tiles(cells), scan_tiles(count)) + 1;
}

int ingest_make_keys(const LaunchCfg& c, cudaStream_t s, const int32_t* src, const int32_t* dst,
                     int64_t m, int64_t n, int B, int directed, unsigned long long* keys, int* bad) {
  if (m <= 0) return 0;
  k_make_keys<<<c.grid, c.block, 0, s>>>(src, dst, m, n, B, directed, keys, bad);
  return 1;
}

int ingest_swap_keys(const LaunchCfg& c, cudaStream_t s, const unsigned long long* in, int64_t count,
                     int B, unsigned long long* out) {
  if (count <= 0) return 0;
  k_swap_keys<<<c.grid, c.block, 0, s>>>(in, count, B, out);
  return 1;
}

int radix_sort(cudaStream_t s, unsigned long long*& keys, unsigned long long*& alt, int64_t count,
               int bit0, int bits, int64_t* scratch) {
  if (count <= 1) return 0;
  const int items = rs_items(count);
  const int64_t tiles = rs_tiles(count), cells = 256 * tiles;
  int64_t* off = scratch;
  uint32_t* hist = reinterpret_cast<uint32_t*>(scratch + cells);
  int64_t* sums = scratch + cells + cells / 2;
  int launches = 0;
  for (int shift = bit0; shift < bits; shift += 8) {
    k_rs_hist<<<static_cast<unsigned>(tiles), kRsThreads, 0, s>>>(keys, count, shift, items, tiles, hist);
    if (cells <= kScanShort) {
      k_scan_short<<<1, kScanThreads, 0, s>>>(hist, static_cast<int>(cells), off);
      launches += 1;
    } else {
      const unsigned st = static_cast<unsigned>(scan_tiles(cells));
      k_scan_sums<<<st, kScanThreads, 0, s>>>(Cells{hist}, cells, sums);
      k_scan_sums_excl<<<1, kScanThreads, 0, s>>>(sums, st, nullptr);
      k_scan_out<<<st, kScanThreads, 0, s>>>(Cells{hist}, cells, sums, StorePrefix{off});
      launches += 3;
    }
    k_rs_scatter<<<static_cast<unsigned>(tiles), kRsThreads, 0, s>>>(keys, count, shift, items, tiles, off,
                                                                     alt);
    launches += 2;
    unsigned long long* t = keys;
    keys = alt;
    alt = t;
  }
  return launches;
}

int ingest_count(cudaStream_t s, const unsigned long long* keys, int64_t count, int64_t* scratch, int64_t* nkept) {
  if (count <= 0) return 0;
  const int64_t tiles = scan_tiles(count);
  k_scan_sums<<<static_cast<unsigned>(tiles), kScanThreads, 0, s>>>(FirstCopies{keys}, count, scratch);
  k_scan_sums_excl<<<1, kScanThreads, 0, s>>>(scratch, tiles, nkept);
  return 2;
}

int ingest_emit(cudaStream_t s, const unsigned long long* keys, int64_t count, const int64_t* scratch, int B,
                int32_t* colidx, unsigned long long* kept) {
  if (count <= 0) return 0;
  k_scan_out<<<static_cast<unsigned>(scan_tiles(count)), kScanThreads, 0, s>>>(
      FirstCopies{keys}, count, scratch, EmitArc{keys, (1ull << B) - 1ull, colidx, kept});
  return 1;
}

int ingest_columns(const LaunchCfg& c, cudaStream_t s, const unsigned long long* keys, int64_t count, int B,
                   int32_t* colidx) {
  if (count <= 0) return 0;
  k_columns<<<c.grid, c.block, 0, s>>>(keys, count, B, colidx);
  return 1;
}

int ingest_rows(const LaunchCfg& c, cudaStream_t s, const unsigned long long* keys, int64_t count, int64_t n,
                int B, int64_t* rowptr) {
  k_rows<<<c.grid, c.block, 0, s>>>(keys, count, n, B, rowptr);
  return 1;
}

}  // namespace lgbc
