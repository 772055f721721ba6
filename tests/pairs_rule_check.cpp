// TVAP_OPT_COMPLEX_PAIRS: 0 is none, k > 0 every contraction length from k on; a new context has 81.
#include <math.h>

#include <cstdio>

#include "tvap_internal.cuh"

int main() {
  int bad = 0;
  for (int K = 1; K < 4000; ++K) {
    bad += tvap::complex_pairs(K, 0);
    for (int k : {1, 80, 81, 82, 4000}) bad += tvap::complex_pairs(K, k) != (K >= k);
  }
  const tvap_ctx fresh{};
  bad += fresh.tune_pairs_k != 81;
  std::printf("bad %d\n", bad);
  return bad != 0;
}
