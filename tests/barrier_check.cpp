// Host harness for the waiting rule of lightgraphs.jl_gb300/csrc/grid_barrier.cuh
// (compiled by tests/test_grid_barrier_host.py with g++).  A waiting block is
// played against workers that beat every `gap` polls and stop after `last`;
// prints the poll at which it gives up, or 0 if it has not by `polls`.
#include <cstdio>
#include "grid_barrier.cuh"

using namespace lgbc;

int main() {
  unsigned long long polls, gap, last;
  std::printf("%u %u %u\n", kBarrierPolls, kBeatTurns, kBeatEntries);
  while (std::scanf("%llu %llu %llu", &polls, &gap, &last) == 3) {
    BarrierWait wait;
    unsigned long long up = 0;
    for (unsigned long long p = 1; p <= polls && !up; ++p) {
      const unsigned long long worked = p < last ? p : last;
      if (wait.look() && wait.stuck(gap ? static_cast<unsigned>(worked / gap) : 0u)) up = p;
    }
    std::printf("%llu\n", up);
  }
  BarrierBeat turns, entries;
  unsigned beats = 0;
  for (unsigned turn = 0; turn < 10 * kBeatTurns; ++turn) beats += turns.turn_due() ? 1u : 0u;
  for (unsigned entry = 0; entry < 10 * kBeatEntries; ++entry) beats += entries.entry_due() ? 1u : 0u;
  BarrierBeat rows;  // units of 1 and of several beats' worth
  for (unsigned row = 0; row < 10 * kBeatTurns; ++row) beats += rows.work_due(row % 8 == 0 ? 4 * kBeatTurns : 0u) ? 1u : 0u;
  std::printf("%u\n", beats);
  return 0;
}
