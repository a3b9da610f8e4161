// Host harness for the packed terms of lightgraphs.jl_gb300/csrc/xf64.cuh
// (compiled by tests/test_packed_terms_host.py with g++).  Per line
// "n m1 e1 .. mn en" it packs the n values {m, e}, sums them as the gathers do
// and prints the packed words followed by the sum as "m e".
#include <cstdio>
#include "xf64.cuh"

using namespace lgbc;

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    xg64 g = xg_zero();
    for (int i = 0; i < n; ++i) {
      unsigned long long m;
      int e;
      std::scanf("%llu %d", &m, &e);
      const uint64_t w = xg_pack(xf64{m, e});
      std::printf("%llu ", static_cast<unsigned long long>(w));
      if (i % 32 == 0) xg_norm(g);
      xg_add_packed(g, w, i & 1);
    }
    xg_norm(g);
    const xf64 r = xg_packed_sum(g);
    std::printf("%llu %d\n", static_cast<unsigned long long>(r.m), r.e);
  }
  return 0;
}
