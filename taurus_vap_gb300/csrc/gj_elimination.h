// The elimination product of a Gauss-Jordan panel of the Thouless solve, as
// its arguments (host code; tests/gj_elimination_check.cpp compares what it
// reads with what it writes).
#pragma once

#include "tvap_internal.cuh"

namespace tvap {

// Columns [c0, c1) of the augmented systems W (n x 2n, column-major, one per
// batch entry) after the panel of columns [j0, j0 + nbp): every row but the
// block rows j0 .. j0 + nbp - 1 loses W[:, panel] R, R = the block rows.
// C runs over all rows, so it contains R: the block rows (their panel entries
// are zeros) are kept, else CTAs of a kernel on the FP64 pipe would rewrite
// them while others still read them as R, and an infinite R would become NaN.
inline GemmArgs gj_elimination(int n, int j0, int nbp, int c0, int c1, int batch, double2* W) {
  const long long bs = 2LL * n * n;
  GemmArgs g{};
  g.M = n;
  g.N = c1 - c0;
  g.K = nbp;
  g.batch = batch;
  g.A = View{W + size_t(j0) * n, 1, n, bs};
  g.B = View{W + j0 + size_t(c0) * n, 1, n, bs};
  g.C = W + size_t(c0) * n;
  g.crs = 1;
  g.ccs = n;
  g.cbs = bs;
  g.alpha = make_double2(-1.0, 0.0);
  g.beta = make_double2(1.0, 0.0);
  g.three_m = true;
  g.keep0 = j0;
  g.keep_rows = nbp;
  return g;
}

}  // namespace tvap
