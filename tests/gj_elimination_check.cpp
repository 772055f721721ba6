// What the elimination product of a Gauss-Jordan panel reads and what it writes, element by element: the two are
// disjoint, and every row but the block rows is written once.  Prints the number of violations.
#include <math.h>

#include <cstdio>
#include <vector>

#include "gj_elimination.h"

using namespace tvap;

static long long check(int n, int j0, int nbp, int c0, int c1) {
  const int batch = 2;
  std::vector<double2> W(size_t(batch) * 2 * n * n);
  const GemmArgs g = gj_elimination(n, j0, nbp, c0, c1, batch, W.data());
  std::vector<char> read(W.size(), 0), written(W.size(), 0);
  long long bad = 0;
  auto at = [&](const void* p, long long off) { return size_t(static_cast<const double2*>(p) - W.data() + off); };
  for (int b = 0; b < batch; ++b) {
    for (int k = 0; k < g.K; ++k) {
      for (int i = 0; i < g.M; ++i) read[at(g.A.p, i * g.A.rs + k * g.A.cs + b * g.A.bs)] = 1;
      for (int j = 0; j < g.N; ++j) read[at(g.B.p, k * g.B.rs + j * g.B.cs + b * g.B.bs)] = 1;
    }
    for (int i = 0; i < g.M; ++i)
      for (int j = 0; j < g.N; ++j)
        if (g.writes_row(i)) ++written[at(g.C, i * g.crs + j * g.ccs + b * g.cbs)];
  }
  for (size_t e = 0; e < W.size(); ++e) {
    const int r = int(e % n), c = int(e / n % (2 * n));
    const bool block_row = r >= j0 && r < j0 + nbp, column = c >= c0 && c < c1;
    bad += read[e] && written[e];
    bad += written[e] != (column && !block_row ? 1 : 0);
  }
  return bad;
}

int main() {
  long long bad = 0;
  for (int n : {2, 8, 24, 40, 60})
    for (int nb : {2, 7, 28, 32})
      for (int j0 = 0; j0 < n; j0 += nb) {
        const int nbp = nb < n - j0 ? nb : n - j0, j1 = j0 + nbp, j2 = j1 + (nb < n - j1 ? nb : n - j1);
        bad += check(n, j0, nbp, j1, 2 * n) + check(n, j0, nbp, j1, j2) + check(n, j0, nbp, j2, 2 * n);
      }
  GemmArgs plain{};  // a product that keeps no rows writes them all
  for (int i = 0; i < 600; ++i) bad += !plain.writes_row(i);
  std::printf("bad %lld\n", bad);
  return bad != 0;
}
