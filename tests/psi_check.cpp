// Host harness for the two-word psi of lightgraphs.jl_gb300/csrc/xf64.cuh
// (compiled by tests/test_psi_terms_host.py with g++).  Per line
// "n m1 e1 .. mn en" it packs the n values {m, e}, sums them as the
// shared-memory sweeps do and prints the words followed by the sum as "m e".
#include <cstdio>
#include "xf64.cuh"

using namespace lgbc;

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    PsiSum s{0ull, 0};
    for (int i = 0; i < n; ++i) {
      unsigned long long m;
      int e;
      std::scanf("%llu %d", &m, &e);
      const uint64_t w = psi_pack(xf64{m, e});
      std::printf("%llu ", static_cast<unsigned long long>(w));
      psi_add(s, static_cast<uint32_t>(w), static_cast<uint32_t>(w >> 32), (i & 1) != 0);
      psi_add(s, 0u, 0u, (i & 1) == 0);  // a neighbour that is no successor
      if (i % 32 == 31) psi_norm(s);
    }
    const xf64 r = psi_value(s);
    std::printf("%llu %d\n", static_cast<unsigned long long>(r.m), r.e);
  }
  return 0;
}
