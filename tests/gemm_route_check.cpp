// small_product against measured times (us, cold caches) of both sides, shapes over its range whose sides differ by a
// quarter or more: it takes the faster one.  Prints the number of shapes it gets wrong.
#include <cstdio>

#include "gemm_route.h"

using namespace tvap;

struct Shape {
  int parts, M, N, K, batch;
  Route other;
  double small_us, other_us;
};
static const Shape kShapes[] = {
    {2, 34, 34, 8, 16, Route::fp64_tiles, 7.8, 9.9},
    {2, 137, 137, 8, 1, Route::fp64_tiles, 7.8, 10.5},
    {3, 112, 112, 8, 1, Route::fp64_tiles, 7.8, 11.9},
    {1, 81, 81, 8, 57, Route::fp64_tiles, 22.1, 16.0},
    {1, 187, 187, 3, 57, Route::fp64_tiles, 63.4, 24.2},
    {1, 1414, 1414, 3, 1, Route::fp64_tiles, 60.1, 24.2},
    {1, 1055, 66, 3, 57, Route::fp64_tiles, 126.6, 46.7},
    {2, 1725, 108, 8, 4, Route::fp64_tiles, 55.6, 36.4},
    {3, 1150, 1150, 3, 1, Route::fp64_tiles, 110.8, 51.5},
    {1, 140, 140, 140, 1, Route::mma_sync, 15.6, 27.0},
    {3, 120, 7, 70, 16, Route::tcgen05, 18.1, 26.9},
    {2, 11, 11, 70, 57, Route::tcgen05, 14.0, 25.2},
    {1, 100, 6, 28, 57, Route::tcgen05, 9.8, 22.8},
    {3, 632, 40, 40, 1, Route::tcgen05, 16.0, 25.2},
    {2, 103, 103, 140, 4, Route::tcgen05, 37.1, 26.9},
    {2, 461, 461, 28, 1, Route::tcgen05, 39.1, 24.8},
    {2, 610, 610, 16, 1, Route::tcgen05, 42.3, 23.2},
    {2, 122, 8, 40, 4, Route::mma_sync, 9.9, 23.2},
    {1, 110, 7, 1000, 4, Route::mma_sync, 67.9, 127.6},
    {3, 40, 40, 20, 5, Route::mma_sync, 10.6, 23.2},
    {1, 756, 47, 28, 1, Route::mma_sync, 9.8, 19.1},
    {1, 4000, 1, 1000, 1, Route::tcgen05, 89.7, 147.7},
    {1, 2000, 2, 600, 1, Route::tcgen05, 38.5, 49.8},
    {3, 1000, 2, 600, 1, Route::tcgen05, 71.9, 49.4},
    {3, 8000, 4, 100, 1, Route::tcgen05, 65.2, 29.3},
};

int main() {
  int bad = 0;
  for (const Shape& s : kShapes) {
    const bool small = small_product(s.M, s.N, s.K, s.batch, s.parts, false, s.other);
    if (small != (s.small_us < s.other_us)) {
      std::printf("%d %d x %d x %d x %d\n", s.parts, s.M, s.N, s.K, s.batch);
      ++bad;
    }
  }
  // never emulated below 10^6 multiply-adds, a complex one counted once
  for (int parts = 1; parts <= 3; ++parts)
    for (int K = 16; K <= 4096; K *= 2)
      for (int side = 8; double(side) * side * K < 1e6; side += 8)
        bad += !small_product(side, side, K, 1, parts, false, Route::tcgen05);
  // never on the FP64 pipe above the limit; rows beyond the grid of the FP64 tiles
  bad += small_product(300, 300, 140, 1, 1, false, Route::tcgen05);
  bad += !small_product(2000000, 1, 3, 1, 1, false, Route::fp64_tiles);
  std::printf("bad %d\n", bad);
  return bad != 0;
}
