// bfs.cu -- direction-optimising level-synchronous BFS for gdistances.
//
// Replaces gdistances! (src/traversals/bfs.jl:95-124) and its threaded
// variant (src/Parallel/traversals/gdistances.jl:36-116): every source gets
// level 0, every other vertex the level at which the BFS first reaches it,
// INT32_MAX where nothing reaches it.  The per-level sort of the reference
// (bfs.jl:121) only fixes visiting order and does not change any distance.
//
// A handle's search is one cooperative launch (k_bfs_run): one block per SM
// runs every level, with a grid barrier between levels in place of three or
// four launches and a host round trip.  Top-down levels expand the frontier
// queue over out-edges: a warp streams the concatenated out-lists of up to 32
// frontier vertices (fewer when the frontier is small, so that every warp has
// some), and a vertex with more than kBfsChunk out-edges is cut into pieces of
// that many edges which the whole grid shares.  The visited bitmap (n / 8
// bytes) is tested before any atomic.  Bottom-up levels give each unvisited
// vertex one thread that scans its in-edges and stops at the first
// in-neighbour in the frontier bitmap, staged in shared memory when it fits; a
// warp owns 32 consecutive vertices, hence one word of the visited and next
// bitmaps, and needs no atomics at all: the queue of the new frontier is only
// built when the next level goes top-down.
// Bound: latency of the barriers and of dependent loads on the small levels
// (5 to 10 us a level), in-edge sectors from HBM on the bottom-up ones.  A
// single-source call on R-MAT 20, 4 MB of distances included, takes 139 us
// (226 us with one edge per thread in flight and every warp reading the
// level's counters; host-driven levels more than 400 us).
//
// The kernels with one launch per level serve lgbc_gdistances_noalloc, whose
// fixed scratch holds a queue and two bitmaps.
#include <algorithm>

#include "lgbc_kernels.h"

namespace lgbc {
namespace {

__device__ __forceinline__ long long gwarp() {
  return (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
}
__device__ __forceinline__ long long nwarps() {
  return (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
}

__device__ __forceinline__ unsigned long long shfl_up_u64(unsigned long long x, int o) {
  const unsigned lo = __shfl_up_sync(kFull, static_cast<unsigned>(x), o);
  const unsigned hi = __shfl_up_sync(kFull, static_cast<unsigned>(x >> 32), o);
  return (static_cast<unsigned long long>(hi) << 32) | lo;
}

__device__ __forceinline__ int64_t shfl_i64(int64_t x, int src) {
  return static_cast<int64_t>(shfl_u64(static_cast<uint64_t>(x), src));
}

__device__ __forceinline__ uint32_t* bm_at(const BfsBuffers& b, int level) {
  return (level & 1) ? b.bm[1] : b.bm[0];
}

__global__ void k_bfs_ctl_reset(BatchCtl* c) {
  c->lo = 0;
  c->hi = 0;
  c->tail = 0;
  c->mf = 0;
  c->mf_cur = 0;
  c->mu_done = 0;
  c->cap = 0;
  c->level = 0;
  c->maxlevel = 0;
  c->done = 0;
  c->overflow_list = 0;
  c->overflow_sigma = 0;
  c->mode = 0;
}

// Level 0: claim each source once (duplicates in the source list are
// harmless, as in bfs.jl:103-107).
__global__ void k_bfs_seed(DevGraph g, BfsBuffers b, const int32_t* src, int64_t nsrc,
                           int32_t* dist) {
  BatchCtl* c = b.ctl;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nsrc;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t s = src[i];
    if (atomicCAS(dist + s, kUnreached, 0) == kUnreached) {
      const unsigned long long slot = atomicAdd(&c->tail, 1ull);
      b.queue[slot] = s;
      atomicOr(&b.bm[0][s >> 5], 1u << (s & 31));
      atomicAdd(&c->mf, static_cast<unsigned long long>(g.rowptr[s + 1] - g.rowptr[s]));
      atomicAdd(&c->mu_done,
                static_cast<unsigned long long>(g.in_rowptr[s + 1] - g.in_rowptr[s]));
    }
  }
}

__global__ void k_bfs_seed_done(BatchCtl* c) {
  c->lo = 0;
  c->hi = c->tail;
  c->mf_cur = c->mf;
  c->mf = 0;
  if (c->tail == 0) {
    c->done = 1;
    c->maxlevel = -1;
  }
}

// Zero the bitmap that the coming top-down level fills with atomicOr.
__global__ void k_bfs_clear_next(BfsBuffers b, int64_t nwords) {
  uint32_t* nbm = bm_at(b, b.ctl->level + 1);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nwords;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    nbm[i] = 0u;
}

// Claim w for level nl if no one has; returns whether this thread did.
__device__ __forceinline__ bool bfs_claim(const DevGraph& g, uint32_t* nbm, int32_t* dist,
                                          int32_t w, int32_t nl, unsigned long long& mf,
                                          unsigned long long& mu) {
  if (dist[w] != kUnreached || atomicCAS(dist + w, kUnreached, nl) != kUnreached) return false;
  atomicOr(nbm + (w >> 5), 1u << (w & 31));
  mf += static_cast<unsigned long long>(g.rowptr[w + 1] - g.rowptr[w]);
  mu += static_cast<unsigned long long>(g.in_rowptr[w + 1] - g.in_rowptr[w]);
  return true;
}

__device__ __forceinline__ void bfs_flush_counts(BatchCtl* c, unsigned long long mf,
                                                 unsigned long long mu) {
  mf = warp_sum_u64(mf);
  mu = warp_sum_u64(mu);
  if (lane_id() == 0) {
    if (mf) atomicAdd(&c->mf, mf);
    if (mu) atomicAdd(&c->mu_done, mu);
  }
}

// Top-down level: lane j of a warp holds frontier entry base + j.  The 32
// out-lists are walked as one concatenation, edge k of it by lane k % 32 (the
// owning vertex found by a binary search over the warp's inclusive degree
// scan).
__global__ void __launch_bounds__(256) k_bfs_td(DevGraph g, BfsBuffers b, int32_t* dist) {
  BatchCtl* c = b.ctl;
  const unsigned long long lo = c->lo, hi = c->hi;
  const int32_t nl = c->level + 1;
  uint32_t* nbm = bm_at(b, nl);
  const int ln = lane_id();
  unsigned long long mf = 0, mu = 0;
  for (unsigned long long base = lo + static_cast<unsigned long long>(gwarp()) * kWarp; base < hi;
       base += static_cast<unsigned long long>(nwarps()) * kWarp) {
    const unsigned long long i = base + ln;
    int32_t v = 0;
    int64_t e0 = 0, deg = 0;
    if (i < hi) {
      v = b.queue[i];
      e0 = g.rowptr[v];
      deg = g.rowptr[v + 1] - e0;
    }
    const int d = static_cast<int>(deg);
    int incl = d;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (ln >= o) incl += y;
    }
    const int total = __shfl_sync(kFull, incl, kWarp - 1);
    const int off = incl - d;
    for (int k0 = 0; k0 < total; k0 += kWarp) {
      const int k = k0 + ln;
      int j = 0;  // the lane whose list holds concatenated edge k: the first with incl > k
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1) {
        const int iv = __shfl_sync(kFull, incl, j + step - 1);
        if (iv <= k) j += step;
      }
      const int64_t ej = shfl_i64(e0, j);
      const int oj = __shfl_sync(kFull, off, j);
      bool app = false;
      int32_t w = 0;
      if (k < total) {
        w = g.colidx[ej + (k - oj)];
        app = bfs_claim(g, nbm, dist, w, nl, mf, mu);
      }
      const unsigned long long q = warp_append(app, &c->tail);
      if (app) b.queue[q] = w;
    }
  }
  bfs_flush_counts(c, mf, mu);
}

template <bool STAGE>
__global__ void __launch_bounds__(1024) k_bfs_bu(DevGraph g, BfsBuffers b, int32_t* dist) {
  extern __shared__ uint32_t sbm[];
  BatchCtl* c = b.ctl;
  const int32_t nl = c->level + 1;
  const int64_t n = g.n;
  const int64_t nwords = (n + 31) >> 5;
  const uint32_t* fbm = bm_at(b, nl - 1);
  uint32_t* nbm = bm_at(b, nl);
  if (STAGE) {
    const uint4* src4 = reinterpret_cast<const uint4*>(fbm);
    uint4* dst4 = reinterpret_cast<uint4*>(sbm);
    const int64_t n4 = nwords >> 2;
    for (int64_t i = threadIdx.x; i < n4; i += blockDim.x) dst4[i] = src4[i];
    for (int64_t i = (n4 << 2) + threadIdx.x; i < nwords; i += blockDim.x) sbm[i] = fbm[i];
    __syncthreads();
    fbm = sbm;
  }
  const int ln = lane_id();
  unsigned long long mf = 0, mu = 0;
  for (int64_t base = gwarp() * kWarp; base < n; base += nwarps() * kWarp) {
    const int64_t w = base + ln;
    bool found = false;
    if (w < n && dist[w] == kUnreached) {
      const int64_t e1 = g.in_rowptr[w + 1];
      for (int64_t e = g.in_rowptr[w]; e < e1; ++e) {
        const int32_t v = g.in_colidx[e];
        if ((fbm[v >> 5] >> (v & 31)) & 1u) {
          found = true;
          break;
        }
      }
    }
    const unsigned bal = __ballot_sync(kFull, found);
    if (ln == 0) nbm[base >> 5] = bal;
    if (found) {
      dist[w] = nl;
      mf += static_cast<unsigned long long>(g.rowptr[w + 1] - g.rowptr[w]);
      mu += static_cast<unsigned long long>(g.in_rowptr[w + 1] - g.in_rowptr[w]);
    }
    const unsigned long long slot = warp_append(found, &c->tail);
    if (found) b.queue[slot] = static_cast<int32_t>(w);
  }
  mf = warp_sum_u64(mf);
  mu = warp_sum_u64(mu);
  if (ln == 0) {
    if (mf) atomicAdd(&c->mf, mf);
    if (mu) atomicAdd(&c->mu_done, mu);
  }
}

__global__ void k_bfs_advance(BatchCtl* c) {
  if (c->tail == c->hi) {
    c->done = 1;
    c->maxlevel = c->level;
    c->mf_cur = 0;
    return;
  }
  c->lo = c->hi;
  c->hi = c->tail;
  c->level += 1;
  c->mf_cur = c->mf;
  c->mf = 0;
}

// ---------------------------------------------------------------------------
// The whole search in one cooperative launch.
// ---------------------------------------------------------------------------

// What a thread has found in this level.
struct BfsFound {
  unsigned count = 0;
  unsigned long long mf = 0, mu = 0;
};

// List the vertices w[q] where ok[q], with rows of d[q] entries, for a level
// of the given parity: one atomic per warp for the queue and one for the long
// rows.  That one hands out entries (high word) and their first chunks (low
// word), so the list is sorted by first chunk; an atomic for every long row
// was 1.4 ns each on the one address, and neighbours of hubs are often hubs.
template <int Q>
__device__ __forceinline__ void bfs_append(const BfsRun& r, BfsSlot* slot, unsigned long long base, int parity,
                                           const int32_t (&w)[Q], const int64_t (&d)[Q], const bool (&ok)[Q]) {
  const int ln = lane_id();
  int at[Q], total = 0;
  unsigned long long mine = 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const unsigned bal = __ballot_sync(kFull, ok[q] && d[q] <= kBfsChunk);
    at[q] = total + __popc(bal & ((1u << ln) - 1u));
    total += __popc(bal);
    if (ok[q] && d[q] > kBfsChunk) mine += (1ull << 32) | static_cast<unsigned>((d[q] + kBfsChunk - 1) / kBfsChunk);
  }
  unsigned long long first = 0;
  if (ln == 0 && total) first = atomicAdd(&slot->queued, static_cast<unsigned long long>(total));
  const bool big = __any_sync(kFull, mine != 0ull);
  unsigned long long p = mine;
  if (big) {
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const unsigned long long y = shfl_up_u64(p, o);
      if (ln >= o) p += y;
    }
    unsigned long long b0 = 0;
    if (ln == kWarp - 1) b0 = atomicAdd(&slot->big, p);
    p = static_cast<unsigned long long>(shfl_i64(static_cast<int64_t>(b0), kWarp - 1)) + p - mine;
  }
  first = base + static_cast<unsigned long long>(shfl_i64(static_cast<int64_t>(first), 0));
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!ok[q]) continue;
    if (d[q] <= kBfsChunk) {
      r.queue[first + at[q]] = w[q];
    } else {
      r.big[parity * r.big_cap + static_cast<int64_t>(p >> 32)] = make_int2(static_cast<int>(p & 0xFFFFFFFFu), w[q]);
      p += (1ull << 32) | static_cast<unsigned>((d[q] + kBfsChunk - 1) / kBfsChunk);
    }
  }
}

// List w (claimed by this thread) for a level.
__device__ __forceinline__ void bfs_list(const DevGraph& g, const BfsRun& r, BfsSlot* slot,
                                         unsigned long long base, int parity, bool claimed, int32_t w,
                                         BfsFound& f) {
  int64_t d = 0;
  if (claimed) {
    d = g.rowptr[w + 1] - g.rowptr[w];
    f.count += 1;
    f.mf += static_cast<unsigned long long>(d);
    f.mu += static_cast<unsigned long long>(g.in_rowptr[w + 1] - g.in_rowptr[w]);
  }
  const int32_t ws[1] = {w};
  const int64_t ds[1] = {d};
  const bool oks[1] = {claimed};
  bfs_append<1>(r, slot, base, parity, ws, ds, oks);
}

// Take the edges to w[q] where ok[q] for level `level` and list what they
// reach.  Every step of the chain (visited word, claim, row lengths, queue
// entry) is a round trip of about a microsecond, so kBfsAhead edges per thread
// go through it together, with one queue atomic for all of the warp's.
__device__ __forceinline__ void bfs_expand(const DevGraph& g, const BfsRun& r, uint32_t* next, BfsSlot* slot,
                                           unsigned long long base, int32_t level, const int32_t (&w)[kBfsAhead],
                                           bool (&ok)[kBfsAhead], BfsFound& f) {
  uint32_t word[kBfsAhead];
#pragma unroll
  for (int q = 0; q < kBfsAhead; ++q)  // a stale cached word can only lack bits, which the atomic then finds set
    word[q] = ok[q] ? r.visited[w[q] >> 5] : ~0u;
#pragma unroll
  for (int q = 0; q < kBfsAhead; ++q) {
    const uint32_t bit = 1u << (w[q] & 31);
    if (!(word[q] & bit)) word[q] = atomicOr(r.visited + (w[q] >> 5), bit);
  }
  bool any = false;
#pragma unroll
  for (int q = 0; q < kBfsAhead; ++q) {
    const uint32_t bit = 1u << (w[q] & 31);
    ok[q] = !(word[q] & bit);
    any |= ok[q];
    if (ok[q]) {
      atomicOr(next + (w[q] >> 5), bit);
      r.dist[w[q]] = level;
    }
  }
  if (!__any_sync(kFull, any)) return;
  int64_t d[kBfsAhead];
#pragma unroll
  for (int q = 0; q < kBfsAhead; ++q) {
    d[q] = 0;
    if (ok[q]) {
      d[q] = g.rowptr[w[q] + 1] - g.rowptr[w[q]];
      f.mu += static_cast<unsigned long long>(g.in_rowptr[w[q] + 1] - g.in_rowptr[w[q]]);
    }
  }
#pragma unroll
  for (int q = 0; q < kBfsAhead; ++q) {
    f.count += ok[q] ? 1u : 0u;
    f.mf += static_cast<unsigned long long>(d[q]);
  }
  bfs_append<kBfsAhead>(r, slot, base, level & 1, w, d, ok);
}

__global__ void __launch_bounds__(1024, 1) k_bfs_run(DevGraph g, BfsRun r) {
  extern __shared__ uint32_t sbm[];
  __shared__ int s_ok, s_bu;
  __shared__ unsigned long long s_queued, s_big;
  __shared__ unsigned long long s_sum[3];
  BfsState* st = r.state;
  const int ln = lane_id();
  const int64_t n = g.n, nwords = (n + 31) >> 5;
  const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t threads = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const long long warp = gwarp(), warps = nwarps();
  unsigned long long goal = 0;
  BarrierBeat beat, walked;
  auto bitmap = [&](int32_t level) { return r.visited + (1 + level % 3) * r.words; };

  // fold a level's findings into its slot, one set of atomics per block
  auto report = [&](BfsSlot* slot, const BfsFound& f) {
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0ull;
    __syncthreads();
    const unsigned c = __reduce_add_sync(kFull, f.count);
    const unsigned long long mf = warp_sum_u64(f.mf), mu = warp_sum_u64(f.mu);
    if (ln == 0 && c) {
      atomicAdd(&s_sum[0], static_cast<unsigned long long>(c));
      atomicAdd(&s_sum[1], mf);
      atomicAdd(&s_sum[2], mu);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_sum[0]) {
      atomicAdd(&slot->count, s_sum[0]);
      atomicAdd(&slot->mf, s_sum[1]);
      atomicAdd(&slot->mu, s_sum[2]);
    }
  };

  // distances, bitmaps (prefilled: distances other than kUnreached are
  // vertices the search must leave alone)
  for (int64_t w0 = warp * kWarp; w0 < nwords * kWarp; w0 += warps * kWarp) {
    const int64_t v = w0 + ln;
    bool seen = v >= n;
    if (v < n) {
      if (r.prefilled) seen = r.dist[v] != kUnreached;
      else r.dist[v] = kUnreached;
      // no edge reaches it: else a bottom-up level would come back to it each
      // time (two fifths of an R-MAT graph)
      seen |= g.in_rowptr[v + 1] == g.in_rowptr[v];
    }
    const unsigned bal = __ballot_sync(kFull, seen);
    if (ln == 0) {
      r.visited[w0 >> 5] = bal;
      bitmap(0)[w0 >> 5] = 0u;
      bitmap(1)[w0 >> 5] = 0u;
    }
  }
  if (!grid_barrier(&st->barrier, goal, &s_ok)) return;
  {
    BfsFound f;
    for (int64_t i0 = tid - ln; i0 < r.nsrc; i0 += threads) {
      const int64_t i = i0 + ln;
      const int32_t s = i < r.nsrc ? r.src[i] : 0;
      // by the frontier's bit: a source that nothing enters has its visited bit
      const uint32_t bit = 1u << (s & 31);
      bool claimed = i < r.nsrc && (!r.prefilled || __ldcg(r.dist + s) == kUnreached);
      if (claimed) claimed = !(atomicOr(bitmap(0) + (s >> 5), bit) & bit);
      if (claimed) {
        atomicOr(r.visited + (s >> 5), bit);
        r.dist[s] = 0;
      }
      bfs_list(g, r, &st->slot[0], 0, 0, claimed, s, f);
    }
    report(&st->slot[0], f);
  }
  if (!grid_barrier(&st->barrier, goal, &s_ok)) return;

  unsigned long long lo = 0, mu_done = 0;
  bool bu = false;
  long long td_levels = 0, bu_levels = 0;
  for (int32_t level = 0;; ++level) {
    // a slot is reused three levels later, by when every block has read it
    const BfsSlot* cur = &st->slot[level % 3];
    BfsSlot* nxt = &st->slot[(level + 1) % 3];
    // One thread reads the slot and chooses the direction: the reads of every
    // warp went to one L2 line (24,000 of them, 10 us a level), and a division
    // of 1,024 threads keeps the FP64 pipe for some more.
    if (threadIdx.x == 0) {
      const unsigned long long count = __ldcg(&cur->count), mf = __ldcg(&cur->mf);
      s_queued = __ldcg(&cur->queued);
      s_big = __ldcg(&cur->big);
      mu_done += __ldcg(&cur->mu);
      const double left = static_cast<double>(g.nnz) - static_cast<double>(mu_done);
      s_bu = count == 0 ? -1
             : bu       ? static_cast<double>(count) >= static_cast<double>(n) / r.beta
                        : static_cast<double>(mf) > left / r.alpha;
    }
    __syncthreads();
    const bool was = bu;
    if (s_bu < 0 || level > n) break;
    bu = s_bu != 0;
    unsigned long long queued = s_queued, big = s_big;
    uint32_t* front = bitmap(level);
    uint32_t* next = bitmap(level + 1);
    uint32_t* stale = bitmap(level + 2);
    if (was && !bu) {
      // the frontier exists only as a bitmap: list it, in this level's own slot
      BfsSlot* own = &st->slot[level % 3];
      BfsFound ignored;
      for (int64_t w0 = warp * kWarp; w0 < nwords; w0 += warps * kWarp) {
        uint32_t bits = w0 + ln < nwords ? __ldcg(front + w0 + ln) : 0u;
        while (__any_sync(kFull, bits != 0u)) {
          const bool has = bits != 0u;
          const int32_t v = static_cast<int32_t>((w0 + ln) * kWarp + (has ? __ffs(bits) - 1 : 0));
          bits &= bits - 1u;
          bfs_list(g, r, own, lo, level & 1, has, v, ignored);
        }
      }
      if (!grid_barrier(&st->barrier, goal, &s_ok)) return;
      if (threadIdx.x == 0) {
        s_queued = __ldcg(&own->queued);
        s_big = __ldcg(&own->big);
      }
      __syncthreads();
      queued = s_queued;
      big = s_big;
    }
    // what the level after next will fill
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      BfsSlot* z = &st->slot[(level + 2) % 3];
      z->count = z->mf = z->mu = z->queued = z->big = 0ull;
    }
    for (int64_t i = tid; i < nwords; i += threads) stale[i] = 0u;
    const unsigned long long hi = lo + queued;
    BfsFound f;
    if (bu) {
      ++bu_levels;
      const uint32_t* fbm = front;
      if (r.stage) {
        const uint4* src4 = reinterpret_cast<const uint4*>(front);
        uint4* dst4 = reinterpret_cast<uint4*>(sbm);
        // eight loads in flight
        const int64_t quads = (nwords + 3) >> 2;
        for (int64_t i0 = threadIdx.x; i0 < quads; i0 += 8 * blockDim.x) {
          uint4 x[8];
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (i0 + q * blockDim.x < quads) x[q] = __ldcg(src4 + i0 + q * blockDim.x);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (i0 + q * blockDim.x < quads) dst4[i0 + q * blockDim.x] = x[q];
        }
        __syncthreads();
        fbm = sbm;
      }
      // A warp's words are loaded 32 at a time, and a word's row pointers while
      // the rows of the word before are looked through: what is left for a word
      // is its columns' round trips.
      for (int64_t g0 = warp; g0 < nwords; g0 += warps * kWarp) {
        const int64_t mine = g0 + ln * warps;
        const uint32_t words = mine < nwords ? __ldcg(r.visited + mine) : ~0u;
        if (mine < nwords && words == ~0u) next[mine] = 0u;
        unsigned todo = __ballot_sync(kFull, words != ~0u);
        int64_t en = 0, en1 = 0;
        auto rows_of = [&](int k) {
          const int64_t v = ((g0 + k * warps) << 5) + ln;
          en = en1 = 0;
          if (!((__shfl_sync(kFull, words, k) >> ln) & 1u)) {
            en = g.in_rowptr[v];
            en1 = g.in_rowptr[v + 1];
          }
        };
        if (todo) rows_of(__ffs(todo) - 1);
        while (todo) {
          const int k = __ffs(todo) - 1;
          todo &= todo - 1u;
          const int64_t w0 = g0 + k * warps, v = (w0 << 5) + ln;
          const uint32_t seen = __shfl_sync(kFull, words, k);
          int64_t e = en;
          const int64_t e1 = en1;
          const unsigned long long din = static_cast<unsigned long long>(e1 - e);
          if (todo) rows_of(__ffs(todo) - 1);
          bool found = false;
          for (; !found && e < e1; ++e) {
            const int32_t u = g.in_colidx[e];
            const uint32_t word = r.stage ? fbm[u >> 5] : __ldcg(fbm + (u >> 5));
            found = ((word >> (u & 31)) & 1u) != 0u;
            if (walked.entry_due()) beat_now(&st->barrier);
          }
          const unsigned bal = __ballot_sync(kFull, found);
          if (ln == 0) {
            next[w0] = bal;
            if (bal) r.visited[w0] = seen | bal;
          }
          if (found) {
            r.dist[v] = level + 1;
            f.count += 1;
            f.mu += din;
            f.mf += g.rowptr == g.in_rowptr ? din : static_cast<unsigned long long>(g.rowptr[v + 1] - g.rowptr[v]);
          }
        }
      }
    } else {
      ++td_levels;
      // vertices a warp takes at a time: all warps get some
      int per = static_cast<int>((queued + static_cast<unsigned long long>(warps) - 1) /
                                 static_cast<unsigned long long>(warps));
      per = per < 1 ? 1 : (per > kWarp ? kWarp : per);
      for (unsigned long long base = lo + static_cast<unsigned long long>(warp) * per; base < hi;
           base += static_cast<unsigned long long>(warps) * per) {
        const unsigned long long i = base + ln;
        int64_t e0 = 0;
        int d = 0;
        if (ln < per && i < hi) {
          const int32_t v = __ldcg(r.queue + i);
          e0 = g.rowptr[v];
          d = static_cast<int>(g.rowptr[v + 1] - e0);
        }
        int incl = d;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
          const int y = __shfl_up_sync(kFull, incl, o);
          if (ln >= o) incl += y;
        }
        const int total = __shfl_sync(kFull, incl, kWarp - 1);
        const int off = incl - d;
        for (int k0 = 0; k0 < total; k0 += kBfsAhead * kWarp) {
          beat_turn(&st->barrier, beat);
          int32_t w[kBfsAhead];
          bool ok[kBfsAhead];
#pragma unroll
          for (int q = 0; q < kBfsAhead; ++q) {
            const int k = k0 + q * kWarp + ln;
            ok[q] = k < total;
            w[q] = 0;
            if (k0 + q * kWarp >= total) continue;  // warp-uniform
            int j = 0;  // the lane whose list holds concatenated edge k
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
              const int iv = __shfl_sync(kFull, incl, j + step - 1);
              if (iv <= k) j += step;
            }
            const int64_t ej = shfl_i64(e0, j);
            const int oj = __shfl_sync(kFull, off, j);
            if (ok[q]) w[q] = g.colidx[ej + (k - oj)];
          }
          bfs_expand(g, r, next, nxt, hi, level + 1, w, ok, f);
        }
      }
      const long long entries = static_cast<long long>(big >> 32), chunks = static_cast<long long>(big & 0xFFFFFFFFull);
      const int2* list = r.big + (level & 1) * r.big_cap;
      for (long long c = warp; c < chunks; c += warps) {
        beat_turn(&st->barrier, beat);
        long long a = 0, b = entries - 1;  // the last entry whose first chunk is at most c
        while (a < b) {
          const long long mid = (a + b + 1) >> 1;
          if (__ldcg(&list[mid]).x <= c) a = mid;
          else b = mid - 1;
        }
        const int2 en = __ldcg(&list[a]);
        const int64_t e0 = g.rowptr[en.y] + (c - en.x) * kBfsChunk;
        const int64_t e1 = min(e0 + kBfsChunk, g.rowptr[en.y + 1]);
        int32_t w[kBfsAhead];
        bool ok[kBfsAhead];
#pragma unroll
        for (int q = 0; q < kBfsAhead; ++q) {
          const int64_t idx = e0 + q * kWarp + ln;
          ok[q] = idx < e1;
          w[q] = ok[q] ? g.colidx[idx] : 0;
        }
        bfs_expand(g, r, next, nxt, hi, level + 1, w, ok, f);
      }
    }
    report(nxt, f);
    lo = hi;
    if (!grid_barrier(&st->barrier, goal, &s_ok)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->td_levels = td_levels;
    st->bu_levels = bu_levels;
  }
}

// _bfs_parents (src/traversals/bfs.jl:40-66) visits each level in sorted
// vertex order and gives a newly reached vertex the first level vertex that
// lists it, i.e. the smallest in-neighbour one level closer; the source is
// its own parent, unreached vertices get -1 (0 in 1-based ids).  One warp
// per vertex scans its in-list (sorted ascending) for the first neighbour at
// distance d - 1.
__global__ void __launch_bounds__(256) k_bfs_parents(DevGraph g, const int32_t* dist,
                                                     int32_t* parents) {
  const int ln = lane_id();
  for (long long v = gwarp(); v < g.n; v += nwarps()) {
    const int32_t d = dist[v];
    if (d == kUnreached || d <= 0) {
      if (ln == 0) parents[v] = d == 0 ? static_cast<int32_t>(v) : -1;
      continue;
    }
    const int64_t e0 = g.in_rowptr[v], e1 = g.in_rowptr[v + 1];
    int32_t p = -1;
    for (int64_t e = e0; e < e1; e += kWarp) {
      const int64_t idx = e + ln;
      int32_t u = 0;
      bool hit = false;
      if (idx < e1) {
        u = g.in_colidx[idx];
        hit = dist[u] == d - 1;
      }
      const unsigned bal = __ballot_sync(kFull, hit);
      if (bal) {
        p = __shfl_sync(kFull, u, __ffs(bal) - 1);
        break;
      }
    }
    if (ln == 0) parents[v] = p;
  }
}

__global__ void k_scatter_i32(int32_t* p, const int32_t* idx, int64_t count, int32_t value) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < count;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    p[idx[i]] = value;
}

}  // namespace

size_t bfs_configure(size_t max_dyn_smem) {
  cudaFuncSetAttribute(k_bfs_bu<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(max_dyn_smem));
  cudaFuncAttributes fa{};
  size_t room = 0;
  if (cudaFuncGetAttributes(&fa, k_bfs_run) == cudaSuccess && max_dyn_smem > fa.sharedSizeBytes)
    room = max_dyn_smem - fa.sharedSizeBytes;
  cudaFuncSetAttribute(k_bfs_run, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room));
  return room;
}

int bfs_run(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, BfsRun r, size_t room) {
  cudaMemsetAsync(r.state, 0, sizeof(BfsState), s);
  const size_t bytes = static_cast<size_t>((((g.n + 31) >> 5) + 3) & ~int64_t(3)) * 4;
  r.stage = bytes <= room ? 1 : 0;
  DevGraph dg = g;
  void* args[] = {&dg, &r};
  cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_bfs_run), dim3(static_cast<unsigned>(c.sms)), dim3(1024),
                              args, r.stage ? bytes : 0, s);
  return 1;
}

int bfs_init(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
             const int32_t* src, int64_t nsrc, int32_t* dist) {
  const int64_t nwords = (g.n + 31) >> 5;
  cudaMemsetAsync(b.bm[0], 0, static_cast<size_t>(nwords) * 4, s);
  cudaMemsetAsync(b.bm[1], 0, static_cast<size_t>(nwords) * 4, s);
  k_bfs_ctl_reset<<<1, 1, 0, s>>>(b.ctl);
  int launches = 1;
  if (nsrc > 0) {
    const int grid = static_cast<int>(std::min<int64_t>((nsrc + 255) / 256, c.grid));
    k_bfs_seed<<<grid, 256, 0, s>>>(g, b, src, nsrc, dist);
    ++launches;
  }
  k_bfs_seed_done<<<1, 1, 0, s>>>(b.ctl);
  return launches + 1;
}

int bfs_topdown(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
                int32_t* dist) {
  const int64_t nwords = (g.n + 31) >> 5;
  k_bfs_clear_next<<<c.grid, c.block, 0, s>>>(b, nwords);
  k_bfs_td<<<c.grid, c.block, 0, s>>>(g, b, dist);
  return 2;
}

int bfs_bottomup(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const BfsBuffers& b,
                 int32_t* dist, int stage_smem) {
  const int64_t nwords = (g.n + 31) >> 5;
  if (stage_smem) {
    const size_t bytes = static_cast<size_t>((nwords + 3) & ~int64_t(3)) * 4;
    // one resident 1024-thread block per SM: the bitmap is staged once per SM
    k_bfs_bu<true><<<c.sms, 1024, bytes, s>>>(g, b, dist);
  } else {
    k_bfs_bu<false><<<c.grid, c.block, 0, s>>>(g, b, dist);
  }
  return 1;
}

int bfs_parents(const LaunchCfg& c, cudaStream_t s, const DevGraph& g, const int32_t* dist,
                int32_t* parents) {
  k_bfs_parents<<<c.grid, c.block, 0, s>>>(g, dist, parents);
  return 1;
}

int scatter_i32(const LaunchCfg& c, cudaStream_t s, int32_t* p, const int32_t* idx, int64_t count,
                int32_t value) {
  if (count <= 0) return 0;
  k_scatter_i32<<<c.grid, c.block, 0, s>>>(p, idx, count, value);
  return 1;
}

int bfs_advance(cudaStream_t s, const BfsBuffers& b) {
  k_bfs_advance<<<1, 1, 0, s>>>(b.ctl);
  return 1;
}

}  // namespace lgbc
