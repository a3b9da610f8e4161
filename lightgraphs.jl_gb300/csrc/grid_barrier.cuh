// grid_barrier.cuh -- the grid barrier of kernels launched cooperatively.
#pragma once

#include <stdint.h>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace lgbc {

struct GridBarrier {  // zeroed before the launch
  unsigned long long arrived;
  int failed;
  unsigned beat;      // counts work done between two barriers
};

// A waiting block gives up after this many polls without a beat, which is some
// seconds.  Levels have no such bound of their own (one thread may walk an
// in-list of any length, one block a hub's row), so whatever works in a loop
// between two barriers beats as it goes on (BarrierBeat): a wait ends early
// only when nothing moves any more.
constexpr unsigned kBarrierPolls = 1u << 23;

struct BarrierWait {
  unsigned polls = 0, seen = 0;
  // One poll more without success: true at the end of each stretch of polls,
  // when the beat is to be read and given to stuck().
  __host__ __device__ __forceinline__ bool look() { return ++polls > kBarrierPolls; }
  __host__ __device__ __forceinline__ bool stuck(unsigned beat) {
    const bool same = beat == seen;
    seen = beat;
    polls = 0;
    return same;
  }
};

// What a warp or a thread has done since the launch: every kBeatTurns-th turn of
// a loop, and every kBeatEntries-th entry that one thread walks, is told to the
// waiting blocks.  A turn waits for some hundred loads at most, so a beat
// comes every few tens of milliseconds.  (Loops whose turns are few and short for any
// graph do without.)
constexpr unsigned kBeatTurns = 256;
constexpr unsigned kBeatEntries = 4096;

struct BarrierBeat {
  unsigned count = 0;
  __host__ __device__ __forceinline__ bool turn_due() { return (++count & (kBeatTurns - 1u)) == 0u; }
  // A turn that counts for `units`.
  __host__ __device__ __forceinline__ bool work_due(unsigned units) {
    const unsigned before = count / kBeatTurns;
    count += units;
    return count / kBeatTurns != before;
  }
  __host__ __device__ __forceinline__ bool entry_due() { return (++count & (kBeatEntries - 1u)) == 0u; }
};

#ifdef __CUDACC__
__device__ __forceinline__ void beat_now(GridBarrier* st) { atomicAdd(&st->beat, 1u); }
// One turn of a warp-uniform loop.
__device__ __forceinline__ void beat_turn(GridBarrier* st, BarrierBeat& b) {
  if (b.turn_due() && (threadIdx.x & 31u) == 0u) beat_now(st);
}

// Every block adds one to an ever-growing count and waits until all have.  A
// block that gives up, or sees that another has, reports it, and the kernel
// returns.  All blocks are resident (the launch is cooperative).
__device__ __forceinline__ bool grid_barrier(GridBarrier* st, unsigned long long& goal, int* ok) {
  __syncthreads();
  goal += gridDim.x;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&st->arrived, 1ull);
    BarrierWait wait;
    while (*reinterpret_cast<volatile unsigned long long*>(&st->arrived) < goal &&
           *reinterpret_cast<volatile int*>(&st->failed) == 0) {
      if (wait.look() && wait.stuck(*reinterpret_cast<volatile unsigned*>(&st->beat))) atomicExch(&st->failed, 1);
    }
    __threadfence();
    *ok = *reinterpret_cast<volatile int*>(&st->failed) == 0;
  }
  __syncthreads();
  return *ok != 0;
}
#endif

}  // namespace lgbc
