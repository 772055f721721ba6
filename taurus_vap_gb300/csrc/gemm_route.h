// Which products run on the FP64 pipe in 8 x 8 tiles (small_gemm_kernel) in
// every mode (host code; tests/gemm_route_check.cpp compares the rule with
// measured times of both sides).
#pragma once

namespace tvap {

// what a product that is not a small one runs on
enum class Route { fp64_tiles, tcgen05, mma_sync };

// FP64 multiply-adds of a product (a complex one in the 3M form); `parts`: 1
// real, 2 one complex operand, 3 both.
inline double product_work(double M, double N, double K, double batch, int parts) { return M * N * K * batch * parts; }

// Beyond this the FP64 pipe is never the better one.
constexpr double kSmallWork = 1.2e7;

// Both sides' times (us, cold caches), fitted to 1857 shapes of 0.3 to 12
// million multiply-adds (K = 3 to 1800, 1 to 113 products, thin ones too):
//  - small_gemm_kernel: 7 and, whichever is longer, 0.125 ns x (10 + c K) for
//    each of its tiles (staging and store, then the shared-memory reads: c = 1,
//    2.3, 4 for 1, 2, 3 parts) or a thread's chain along K, 42 to 105 ns a k;
//  - the tcgen05 route: 24 (two slicing passes and a product), 50 ns a k and 9 us
//    for a million operand elements;
//  - the mma.sync products: 20, 150 ns a k and 20 us for a million elements;
//  - the FP64 tiles of 16 to 56 (K < 16, or mode 0) have a chain of 0.3 us a k
//    but half the cost per output; a line through the crossings.
// small / other: 140 x 140 x 140 real 16 / 27, 512 x 256 x 28 complex 40 / 23,
// 280 x 280 x 70 real twice 39 / 29, 4000 x 1 x 1000 real 90 / 148, 996 x 996 x 3
// real four times 112 / 43, 120 x 120 x 8 complex 8 / 12.  The line by the
// multiply-adds alone that stood here took the slower side by up to 2.7 times
// (short K, many tiles); this one is 0.90 of it in the geometric mean and takes
// the faster side for 97 % of the shapes whose sides differ by a quarter.
inline bool small_product(double M, double N, double K, double batch, int parts, bool upper_only, Route other) {
  if (product_work(M, N, K, batch, parts) > kSmallWork) return false;
  auto tiles_of = [](double x) { return double((long long)(x + 7) / 8); };
  const double tiles = tiles_of(M) * tiles_of(N) * batch * (upper_only ? 0.5 : 1.0);
  if (other == Route::fp64_tiles) {
    if (M > 65535.0 * 16) return true;  // their grid holds no more rows
    return tiles * (1.0 + 0.02 * K * parts) <= 400.0 * K;
  }
  if (M * N * K * batch < 1e6) return true;  // never emulated
  const double c = parts == 1 ? 1.0 : parts == 2 ? 2.3 : 4.0, chain = parts == 1 ? 0.042 : parts == 2 ? 0.07 : 0.105;
  const double across = 0.125e-3 * tiles * (10.0 + c * K), along = chain * K;
  const double small_us = 7.0 + (across > along ? across : along);
  const double elems = (M + N) * K * batch * (parts > 1 ? 2.0 : 1.0);
  const double other_us =
      other == Route::tcgen05 ? 24.0 + 0.05 * K + 9e-6 * elems : 20.0 + 0.15 * K + 20e-6 * elems;
  return small_us <= other_us;
}

}  // namespace tvap
