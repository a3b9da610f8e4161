// Host harness for the sums of the dependency gathers, with the bias that the
// kernels use (lightgraphs.jl_gb300/csrc/xf64.cuh; compiled by
// tests/test_gather_sums_host.py with g++).  Per line "n m1 e1 .. mn en" it
// packs the n values {m, e}, sums them and prints the largest exponent byte and
// the sum as "m e".
#include <cstdio>
#include "xf64.cuh"

using namespace lgbc;

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    xg64 g = xg_zero();
    unsigned top = 0;
    for (int i = 0; i < n; ++i) {
      unsigned long long m;
      int e;
      std::scanf("%llu %d", &m, &e);
      const uint64_t w = xg_pack(xf64{m, e}, kXgPsiBias);
      if ((w & 255u) > top) top = static_cast<unsigned>(w & 255u);
      if (i % 32 == 0) xg_norm(g);
      xg_add_packed(g, w, i & 1);
    }
    xg_norm(g);
    const xf64 r = xg_packed_sum(g, kXgPsiBias);
    std::printf("%u %llu %d\n", top, static_cast<unsigned long long>(r.m), r.e);
  }
  return 0;
}
