// The Thouless evolution (cholesky_factorization + evolve_wavefunction,
// module_constraints.f90:497-590) in one cooperative launch: S = 1 + Z^T Z =
// L L^T, A1 = U0 + V0 Z, A2 = V0 + U0 Z, U1 = A1 L^{-T}, V1 = A2 L^{-T}.
#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "tvap_internal.cuh"

namespace tvap {

// ---------------------------------------------------------------------------
// Cholesky factorisation of S (lower, L L^T = S; S has n x n + n doubles, the
// last n receive 1 / L_jj) and the evolution solves
// X L^T = A for two n x n matrices A (U1 = A1 L^{-T}, V1 = A2 L^{-T}) in one
// cooperative launch.  GB300's FP64 pipe gives one SM about 2 FMAs per clock,
// so the factorisation is spread over the grid: panels of kCoopNb columns; CTA
// 0 factors each diagonal block, all CTAs solve the panel rows below it and
// apply the trailing update (CTA 0 updating and factoring the next diagonal
// block meanwhile); then one warp per row of A1 / A2 runs the forward
// substitution L x = a, L read through L2 (beyond kNewtonMaxN it does not fit
// shared memory).  Grid-wide barriers between
// the phases are bounded spins (all CTAs are co-resident by the cooperative
// launch); a barrier that gives up raises the status word and every CTA
// returns.
// ---------------------------------------------------------------------------
namespace {

constexpr int kCoopThreads = 256;
constexpr int kCoopNb = 16;
constexpr long long kCoopSpin = 1LL << 21;

// Grid barrier number `gen` (counted up by every thread): bar[0] counts the
// arrivals of all barriers (zeroed before the launch), bar[2] is the abort
// word.  One releasing increment and an acquiring poll: an arrival counter
// that is reset and a generation word cost two L2 round trips more.
__device__ bool coop_barrier(unsigned* bar, unsigned nblocks, unsigned& gen, int* flags) {
  __shared__ int ok_s;
  ++gen;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned seen;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    for (long long it = 0;; ++it) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (seen >= gen * nblocks) break;
      if (it > kCoopSpin || *(volatile unsigned*)&bar[2]) {
        ok = 0;
        break;
      }
      __nanosleep(20);
    }
    if (!ok || *(volatile unsigned*)&bar[2]) {
      if (!*(volatile unsigned*)&bar[2]) atomicOr(flags, DEV_WAIT_TIMEOUT);
      atomicExch(&bar[2], 1u);
      ok = 0;
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// 1 / sqrt(d) for a positive normal d: an FP32 seed (of d's value with the
// mantissa truncated to 23 bits) refined by two Newton-Raphson steps for the
// reciprocal square root, y <- y (3 - d y^2) / 2 (each step doubles the
// correct bits: 2^-22 -> 2^-44 -> FP64 rounding).  The range test, the seed's
// conversions and d / 2 (an exponent decrement) run on the integer pipe, so
// the 6 Newton instructions are all that occupy the FP64 pipe; outside the
// range of seed_range the library routines are used.
__device__ __forceinline__ double rsqrt_newton(double d) {
  if (!seed_range(d)) return 1.0 / sqrt(d);
  double y = seed_f64(rsqrtf(seed_f32(d)));
  const double h = __longlong_as_double(__double_as_longlong(d) - (1LL << 52));  // d / 2, exact
  y = y * fma(-h, y * y, 1.5);
  y = y * fma(-h, y * y, 1.5);
  return y;
}

// Unblocked Cholesky of the nb x nb diagonal block at (j0, j0) of S by the
// whole CTA (kCoopThreads >= kCoopNb^2 threads, one entry of the block each,
// the block in B): per step the pivot's thread forms 1 / sqrt(d), the column
// is scaled by it (as DPBTF2 does) and the trailing entries take
// A_ij -= L_ik L_jk, each entry in the same order as an unblocked
// elimination.  An FP64 warp instruction holds the FP64 unit of its SM
// sub-partition for about 64 cycles on this part: with the block's entries
// spread over all the CTA's warps, a step's update is one instruction on
// every sub-partition instead of up to 15 on one.  The reciprocals go to
// rd[j0 ..] for the solves; sc (2 doubles of shared memory) carries the
// pivot's reciprocal and the failure flag.  Elements written by other CTAs
// are read through L2.  Every thread of the CTA calls it; the result is
// uniform.
__device__ bool coop_factor_diag(int n, double* S, double* rd, int j0, int nb, double (*B)[kCoopNb + 1],
                                 double* sc) {
  static_assert(kCoopThreads >= kCoopNb * kCoopNb, "one thread per entry of the diagonal block");
  const int t = threadIdx.x;
  const int i = t % kCoopNb, j = t / kCoopNb;
  const bool mine = t < kCoopNb * kCoopNb && i < nb && j < nb && i >= j;
  if (mine) B[i][j] = __ldcg(&S[(j0 + i) + size_t(j0 + j) * n]);
  __syncthreads();
  for (int k = 0; k < nb; ++k) {
    if (t == k * kCoopNb + k) {  // the pivot's thread
      const double d = B[k][k];
      if (d > 0.0) {
        const double y = rsqrt_newton(d);
        B[k][k] = d * y;
        rd[j0 + k] = y;
        sc[0] = y;
        sc[1] = 0.0;
      } else {
        sc[1] = 1.0;
      }
    }
    __syncthreads();
    if (sc[1] != 0.0) return false;  // uniform: read by every thread after the barrier
    if (mine && j == k && i > k) B[i][k] *= sc[0];
    __syncthreads();
    if (mine && j > k) B[i][j] = fma(-B[i][k], B[j][k], B[i][j]);
    __syncthreads();
  }
  if (mine) S[(j0 + i) + size_t(j0 + j) * n] = B[i][j];
  return true;
}

// The factorisation and the solves, called by every thread of a co-resident
// grid (coop_barrier with bar and the caller's generation).  X_m = A_m L^{-T}
// for m = 0 (A at A, X at X) and m = 1 (A + a_stride, X + x_stride); with
// Linv != null also L^{-1} (row r of L^{-T} solves for the unit row e_r).
// coop_smem holds the panel rows, then 1 / L_jj.
template <int SLOTS>
__device__ void evolve_by_blocks(int n, double* S, const double* A, long long a_stride, double* X, long long x_stride,
                                 double* Linv, unsigned* bar, unsigned gen, int* flags, int skip_cta,
                                 double* coop_smem) {
  __shared__ double L11[kCoopNb][kCoopNb + 1];
  __shared__ double rdiag[kCoopNb];
  const int t = threadIdx.x, G = gridDim.x, cta = blockIdx.x;
  double* rd = S + size_t(n) * n;  // 1 / L_jj
  if (cta == 0 && !coop_factor_diag(n, S, rd, 0, min(kCoopNb, n), L11, rdiag) && t == 0) {
    atomicOr(flags, DEV_CHOLESKY);
    atomicExch(&bar[2], 1u);
  }
  // test hook: this CTA leaves without arriving, so that the others' bounded
  // waits at the first barrier run out (status DEV_WAIT_TIMEOUT, abort)
  if (cta == skip_cta) return;
  if (!coop_barrier(bar, G, gen, flags)) return;
  for (int j0 = 0;;) {
    const int j1 = min(j0 + kCoopNb, n);
    if (j1 >= n) break;
    const int nbp = j1 - j0, j2 = min(j1 + kCoopNb, n);
    // panel rows below the diagonal block: L21 = S21 L11^{-T}, one warp per
    // row (lane k holds x_k), rows spread over the CTAs so that their FP64
    // work runs on different SMs
    if (j1 + cta < n) {
      for (int idx = t; idx < nbp * nbp; idx += blockDim.x) {
        const int i = idx % nbp, j = idx / nbp;
        if (i >= j) L11[i][j] = __ldcg(&S[(j0 + i) + size_t(j0 + j) * n]);
      }
      if (t < nbp) rdiag[t] = __ldcg(&rd[j0 + t]);
      __syncthreads();
      const int warp = t >> 5, lane = t & 31, warps = blockDim.x >> 5;
      for (int i = j1 + cta + G * warp; i < n; i += G * warps) {
        double xk = (lane < nbp) ? __ldcg(&S[i + size_t(j0 + lane) * n]) : 0.0;
        for (int m = 0; m < nbp; ++m) {
          if (lane == m) xk *= rdiag[m];
          const double xm = __shfl_sync(0xffffffffu, xk, m);
          if (lane > m && lane < nbp) xk = fma(-xm, L11[lane][m], xk);
        }
        if (lane < nbp) S[i + size_t(j0 + lane) * n] = xk;
      }
    }
    if (!coop_barrier(bar, G, gen, flags)) return;
    // trailing update S22 -= L21 L21^T (lower triangle).  CTA 0 takes the
    // next diagonal block (rows and columns j1 .. j2-1) and factors it; the
    // other CTAs take the rest, one column at a time.  The panel rows j1..n-1
    // are staged in shared memory first (independent loads: one L2 round
    // trip instead of one per k).
    double* P = coop_smem;  // (n - j1) x nbp, row-major
    const int prow = n - j1;
    if (cta == 0 || cta - 1 < prow) {
#pragma unroll 4
      for (int idx = t; idx < prow * nbp; idx += blockDim.x) {
        const int k = idx / prow, i = idx - k * prow;
        P[i * kCoopNb + k] = __ldcg(&S[(j1 + i) + size_t(j0 + k) * n]);
      }
      __syncthreads();
    }
    if (cta == 0) {
      const int nb2 = j2 - j1;
      for (int idx = t; idx < nb2 * nb2; idx += blockDim.x) {
        const int i = idx % nb2, j = idx / nb2;
        if (i < j) continue;
        double v = __ldcg(&S[(j1 + i) + size_t(j1 + j) * n]);
        for (int k = 0; k < nbp; ++k) v = fma(-P[i * kCoopNb + k], P[j * kCoopNb + k], v);
        S[(j1 + i) + size_t(j1 + j) * n] = v;
      }
      __syncthreads();
      // (L11 and rdiag are free until the barrier: every CTA reloads them)
      if (!coop_factor_diag(n, S, rd, j1, nb2, L11, rdiag) && t == 0) {
        atomicOr(flags, DEV_CHOLESKY);
        atomicExch(&bar[2], 1u);
      }
    }
    if (cta > 0 || G == 1) {
      const int workers = G > 1 ? G - 1 : 1, w = G > 1 ? cta - 1 : 0;
      for (int j = j1 + w; j < n; j += workers) {
        const double* pj = P + (j - j1) * kCoopNb;
        const int i0 = (j < j2) ? j2 : j;
        for (int i = i0 + t; i < n; i += blockDim.x) {
          const double* pi = P + (i - j1) * kCoopNb;
          double v = __ldcg(&S[i + size_t(j) * n]);
          for (int k = 0; k < nbp; ++k) v = fma(-pi[k], pj[k], v);
          S[i + size_t(j) * n] = v;
        }
      }
    }
    if (!coop_barrier(bar, G, gen, flags)) return;
    j0 = j1;
  }
  // forward substitution L x = a for every row of A1 and A2: one warp per
  // row, rows spread over all CTAs
  const int warps = blockDim.x >> 5, warp = t >> 5, lane = t & 31;
  const int rows = (Linv ? 3 : 2) * n;
  if (cta >= rows) return;
  // S is written by this grid before the last barrier: read through L2, not L1
  double* dinv = coop_smem;
  __syncthreads();
  for (int j = t; j < n; j += blockDim.x) dinv[j] = __ldcg(&rd[j]);
  __syncthreads();
  constexpr int kMaxPerLane = SLOTS;
  for (int r = cta + G * warp; r < rows; r += G * warps) {
    const int mat = r / n, row = r - mat * n;
    const double* a = A + (mat == 1 ? a_stride : 0);
    double* x = X + (mat == 1 ? x_stride : 0);
    double v[kMaxPerLane];
#pragma unroll
    for (int q = 0; q < kMaxPerLane; ++q) {
      const int j = lane + 32 * q;
      if (mat == 2)
        v[q] = j == row ? 1.0 : 0.0;
      else
        v[q] = (j < n) ? __ldcg(&a[row + size_t(j) * n]) : 0.0;
    }
    // columns j in slot qj (a compile-time index once unrolled): the slots
    // below qj are finished, the slots above take every lane, slot qj the
    // lanes above j -- only those FMAs are issued (each an FP64 instruction
    // of about 64 cycles on this part), in the order of an unblocked solve
#pragma unroll
    for (int qj = 0; qj < kMaxPerLane; ++qj) {
      if (32 * qj >= n) break;
      const int jend = min(32 * qj + 32, n);
      for (int j = 32 * qj; j < jend; ++j) {
        const int owner = j & 31;
        const double xj = __shfl_sync(0xffffffffu, v[qj], owner) * dinv[j];
        if (lane == owner) v[qj] = xj;
        const double* lc = S + size_t(j) * n;
        {
          const int jj = lane + 32 * qj;
          if (jj > j && jj < n) v[qj] = fma(-xj, __ldcg(&lc[jj]), v[qj]);
        }
#pragma unroll
        for (int q = qj + 1; q < kMaxPerLane; ++q) {
          if (32 * q >= n) break;
          const int jj = lane + 32 * q;
          if (jj < n) v[q] = fma(-xj, __ldcg(&lc[jj]), v[q]);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kMaxPerLane; ++q) {
      const int j = lane + 32 * q;
      if (j < n) (mat == 2 ? Linv[j + size_t(row) * n] : x[row + size_t(j) * n]) = v[q];
    }
  }
}


// ---------------------------------------------------------------------------
// L^{-1} without the chain of FP64 pivots.  S = 1 + Z^T Z; X0 = L^{-1} in
// FP32 (one CTA, n <= kNewtonMaxN); then Newton steps in FP64 on the residual
// F = X S X^T - 1:  X <- X - Phi(F) X, Phi(F) = the strict lower triangle and
// half the diagonal, which leaves F^2 (1e-6 -> 1e-12 -> rounding).  Every
// step is three triangular products spread over the grid, each bound by one
// load latency, a few FP64 issues per sub-partition and a grid barrier,
// where each of the n pivots of evolve_by_blocks costs a dependent chain of
// FP64 operations (64 cycles each): n = 140 265 us (two product launches and
// the blocks) -> 155 us cold, with L^{-1} (a single-CTA inverse) 1.1 ms -> 155
// us.  The blocks remain for n > kNewtonMaxN
// (beyond the registers of the FP32 stage) and, in the same launch,
// for an S so ill-conditioned that FP32 gives no usable start (or one with
// non-finite entries, whose status they report).
// ---------------------------------------------------------------------------
constexpr int kNewtonMaxN = 224;
constexpr int kNewtonSteps = 6;
// a residual up to which the step from it is the last: (n f)^2 < 1e-15 in
// the worst case; and one above which FP32 was no use
constexpr float kNewtonLast = 1e-10f, kNewtonUsable = 0.05f;

struct EvolveArgs {
  int n, newton, skip_cta;
  const double *Z, *U0, *V0;
  double *S, *A, *X0, *X1, *T, *E;  // S: n^2 + n; A: A1 then A2; X0, X1, T, E: n^2 each (newton only)
  double *U1, *V1, *Linv;           // Linv may be null
  unsigned* bar;                    // arrivals, (free), abort, then the residual of every Newton step
  int* flags;
};

// The FP32 values of doubles and back by their bits (a conversion is an FP64
// operation): a start value for Newton steps, truncated, below the FP32 range
// zero and above it infinite.
__device__ __forceinline__ float start_f32(double v) {
  const unsigned hi = unsigned(__double2hiint(v)), lo = unsigned(__double2loint(v));
  const int e = int((hi >> 20) & 0x7ff) - 1023 + 127;
  const unsigned m = e <= 0 ? 0u : e >= 255 ? 0x7f800000u : (unsigned(e) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
  return __uint_as_float((hi & 0x80000000u) | m);
}
__device__ __forceinline__ double start_f64(float f) {
  const unsigned u = __float_as_uint(f), e = (u >> 23) & 0xffu;
  const unsigned top = e == 0 ? 0u : (e == 255 ? 0x7ffu : e + 896u) << 20;
  return __hiloint2double(int((u & 0x80000000u) | top | (e == 0 ? 0u : (u & 0x7fffffu) >> 3)), e == 0 ? 0 : int(u << 29));
}

// X = L^{-1} (zeros above the diagonal) in FP32 by one CTA: S = M^{-1} D
// M^{-T} by elimination, in place (column k of M takes the place of column k
// of S at step k: below row k, T_ij -= c_i / d u_j with c column k, u_j = c_j
// right of k, M_kj left of it, 1 at k), and L^{-1} = D^{-1/2} M.
//
// Warp w holds the column pairs w, w + 8, ..; a lane rows lane, lane + 32, ..
// (from the column's own 32-row block on: 60 registers at n = 140).  The steps
// are a chain, taken two at a time; a pair of steps is posted (one mbarrier) by
// the warp of its columns as soon as they are up to date, before the warp's
// other columns are, so that the chain is a pair's own update and what the
// pair does to the other columns runs beside it.  n = 140: 78 us with the
// matrix in shared memory, in blocks of 8 columns with three CTA barriers
// each, 48 us so (the steps 32, reading S 9, writing X 8).
constexpr int kF32Ring = 10;     // pairs kept (nine are needed, as in panel_gj_kernel)
constexpr int kF32MaxSlots = 8;  // 256 rows (kNewtonMaxN = 224)

template <int SLOTS>
struct F32Inverse {
  static constexpr int kCols = 4 * SLOTS;  // of a warp: column q = 2 P + e is column 2 (warp + 8 P) + e
  static constexpr int kLd = 64 * SLOTS + 2;
  float a[kCols][SLOTS];  // column q in slots q / 4 ..
  uint64_t* posted;       // one per pair
  float* ring;            // kF32Ring x kLd: columns k and k + 1 below rows k and k + 1, then 1 / d of both
  float* rv;              // n (+ 1): d^{-1/2}
  int n, warp, lane;

  // columns k (even) and k + 1, up to date in t0 and t1 from slot k / 32 = S0 on
  template <int S0>
  __device__ __forceinline__ void post(const float (&t0)[SLOTS], float (&t1)[SLOTS], int k) {
    const float d0 = __shfl_sync(0xffffffffu, t0[S0], k & 31), below = __shfl_sync(0xffffffffu, t0[S0], (k & 31) + 1);
    const float r0 = __fdividef(1.f, d0), m = below * r0;
    float* out = ring + (k / 2 % kF32Ring) * kLd;
#pragma unroll
    for (int s = S0; s < SLOTS; ++s) t1[s] = fmaf(-m, t0[s], t1[s]);
    const float d1 = __shfl_sync(0xffffffffu, t1[S0], (k & 31) + 1);
    const float r1 = k + 1 < n ? __fdividef(1.f, d1) : 0.f;
#pragma unroll
    for (int s = S0; s < SLOTS; ++s) {
      out[lane + 32 * s] = s > S0 || lane > (k & 31) ? t0[s] : 0.f;
      out[32 * SLOTS + lane + 32 * s] = s > S0 || lane > (k & 31) + 1 ? t1[s] : 0.f;
    }
    if (lane == 0) {
      out[64 * SLOTS] = r0;
      out[64 * SLOTS + 1] = r1;
    }
    __syncwarp();
    if (lane == 0) {
      step_post(&posted[k / 2]);
      rv[k] = rsqrtf(d0);
      rv[k + 1] = rsqrtf(d1);
    }
  }
  // the next pair (not needed again before its steps): columns 4 SK + 0, 1 or
  // 2, 3 of its warp, or 4 SK + 4, 5 if it begins the next 32
  template <int SK>
  __device__ __forceinline__ void ahead(const float (&mu0)[SLOTS], const float (&mu1)[SLOTS], const float* c, int kn) {
    float t0[SLOTS], t1[SLOTS];
    const float u00 = c[kn], u01 = c[32 * SLOTS + kn], u10 = c[kn + 1], u11 = c[32 * SLOTS + kn + 1];
    if (kn < 32 * SK + 32) {
      const bool second = kn >= 32 * SK + 16;
#pragma unroll
      for (int s = SK; s < SLOTS; ++s) {
        const float x0 = a[4 * SK][s], y0 = a[4 * SK + 2][s], x1 = a[4 * SK + 1][s], y1 = a[4 * SK + 3][s];
        t0[s] = fmaf(-mu1[s], u01, fmaf(-mu0[s], u00, second ? y0 : x0));
        t1[s] = fmaf(-mu1[s], u11, fmaf(-mu0[s], u10, second ? y1 : x1));
      }
      post<SK>(t0, t1, kn);
    } else if constexpr (SK + 1 < SLOTS) {
#pragma unroll
      for (int s = SK + 1; s < SLOTS; ++s) {
        t0[s] = fmaf(-mu1[s], u01, fmaf(-mu0[s], u00, a[4 * SK + 4][s]));
        t1[s] = fmaf(-mu1[s], u11, fmaf(-mu0[s], u10, a[4 * SK + 5][s]));
      }
      post<SK + 1>(t0, t1, kn);
    }
  }
  // the factors of every column first, without branches, so that their
  // latencies overlap (0: the pair itself, which follows, and the next one,
  // which is done).  m: the multiplier of row k + 1 in step k
  template <int Q, int SK>
  __device__ __forceinline__ void factors(float (&u0)[kCols], float (&u1)[kCols], const float* c, int k, float m) {
    if constexpr (Q < kCols) {
      const int j = 2 * (warp + 8 * (Q / 2)) + Q % 2;
      if constexpr (Q < 4 * SK + 4) {
        u0[Q] = __shfl_sync(0xffffffffu, a[Q][SK], k & 31);
        u1[Q] = fmaf(-m, u0[Q], __shfl_sync(0xffffffffu, a[Q][SK], (k & 31) + 1));
      }
      if constexpr (Q >= 4 * SK) {
        const float right0 = c[j], right1 = c[32 * SLOTS + j];
        const bool done = Q < 4 * SK + 6 && j < k + 4;
        if constexpr (Q < 4 * SK + 4) {
          u0[Q] = j < k ? u0[Q] : done ? 0.f : right0;
          u1[Q] = j < k ? u1[Q] : done ? 0.f : right1;
        } else {
          u0[Q] = done ? 0.f : right0;
          u1[Q] = done ? 0.f : right1;
        }
      }
      factors<Q + 1, SK>(u0, u1, c, k, m);
    }
  }
  template <int Q, int SK>
  __device__ __forceinline__ void columns(const float (&mu0)[SLOTS], const float (&mu1)[SLOTS],
                                          const float (&u0)[kCols], const float (&u1)[kCols]) {
    if constexpr (Q < kCols) {
      constexpr int s0 = Q / 4 > SK ? Q / 4 : SK;
#pragma unroll
      for (int s = s0; s < SLOTS; ++s) a[Q][s] = fmaf(-mu1[s], u1[Q], fmaf(-mu0[s], u0[Q], a[Q][s]));
      columns<Q + 1, SK>(mu0, mu1, u0, u1);
    }
  }
  // columns k and k + 1 of M, in columns Q and Q + 1
  template <int Q, int SK>
  __device__ __forceinline__ void start(const float (&mu0)[SLOTS], const float (&mu1)[SLOTS], int k, float m) {
    if (k >> 4 == Q / 2) {
#pragma unroll
      for (int s = SK; s < SLOTS; ++s) {
        a[Q][s] = s == SK && lane == (k & 31) ? 1.f : fmaf(mu1[s], m, -mu0[s]);
        a[Q + 1][s] = s == SK && lane == (k & 31) + 1 ? 1.f : -mu1[s];
      }
    }
  }
  template <int SK>
  __device__ __forceinline__ bool steps() {
    if constexpr (SK < SLOTS) {
      for (int k = 32 * SK; k < min(32 * SK + 32, n); k += 2) {
        if (!step_wait(&posted[k / 2])) return false;
        const float* c = ring + (k / 2 % kF32Ring) * kLd;
        const float r0 = c[64 * SLOTS], r1 = c[64 * SLOTS + 1];
        const float m = c[k + 1] * r0;
        float mu0[SLOTS], mu1[SLOTS];
#pragma unroll
        for (int s = SK; s < SLOTS; ++s) {
          mu0[s] = c[lane + 32 * s] * r0;
          mu1[s] = c[32 * SLOTS + lane + 32 * s] * r1;
        }
        if (k + 2 < n && warp == ((k / 2 + 1) & 7)) ahead<SK>(mu0, mu1, c, k + 2);
        float u0[kCols], u1[kCols];
        factors<0, SK>(u0, u1, c, k, m);
        columns<0, SK>(mu0, mu1, u0, u1);
        if (warp == ((k / 2) & 7)) {
          start<4 * SK, SK>(mu0, mu1, k, m);
          start<4 * SK + 2, SK>(mu0, mu1, k, m);
        }
      }
      return steps<SK + 1>();
    }
    return true;
  }
  // between the registers and the matrix in shared memory (column-major, n rows)
  template <int Q, bool LOAD>
  __device__ __forceinline__ void transfer(float* T) {
    if constexpr (Q < kCols) {
      const int j = 2 * (warp + 8 * (Q / 2)) + Q % 2;
#pragma unroll
      for (int s = Q / 4; s < SLOTS; ++s) {
        const int i = lane + 32 * s;
        const bool in = i < n && j < n;
        if (LOAD)
          a[Q][s] = in ? T[i + j * n] : 0.f;
        else if (in)
          T[i + j * n] = a[Q][s];
      }
      transfer<Q + 1, LOAD>(T);
    }
  }
};

template <int SLOTS>
__device__ void inverse_f32(int n, const double* S, double* X, double* sm, int* flags) {
  static_assert(kCoopThreads == 256, "eight warps hold the columns");
  __shared__ int s_late;
  F32Inverse<SLOTS> f;
  f.n = n;
  f.warp = threadIdx.x >> 5;
  f.lane = threadIdx.x & 31;
  f.posted = reinterpret_cast<uint64_t*>(sm);
  f.ring = reinterpret_cast<float*>(f.posted + (n + 1) / 2);
  f.rv = f.ring + kF32Ring * f.kLd;
  float* T = f.rv + n + 1;
  if (threadIdx.x == 0) s_late = 0;
  if (int(threadIdx.x) < (n + 1) / 2) step_init(&f.posted[threadIdx.x]);
  // (through shared memory: the conversions are a short loop, not an instance
  // for every register -- a call finds its instructions far away)
  constexpr int kLoads = 4;
#pragma unroll 1
  for (int j = f.warp; j < n; j += 8 * kLoads) {
    double v[kLoads][SLOTS];
#pragma unroll
    for (int q = 0; q < kLoads; ++q)
#pragma unroll
      for (int s = 0; s < SLOTS; ++s)
        v[q][s] = __ldcg(&S[min(f.lane + 32 * s, n - 1) + min(j + 8 * q, n - 1) * n]);
#pragma unroll
    for (int q = 0; q < kLoads; ++q)
#pragma unroll
      for (int s = 0; s < SLOTS; ++s)
        if (f.lane + 32 * s < n && j + 8 * q < n) T[f.lane + 32 * s + (j + 8 * q) * n] = start_f32(v[q][s]);
  }
  __syncthreads();
  f.template transfer<0, true>(T);
  if (f.warp == 0) f.template post<0>(f.a[0], f.a[1], 0);
  if (!f.template steps<0>()) s_late = 1;
  __syncthreads();
  if (s_late && threadIdx.x == 0) atomicOr(flags, DEV_WAIT_TIMEOUT);
  f.template transfer<0, false>(T);
  __syncthreads();
#pragma unroll 1
  for (int j = f.warp; j < n; j += 8)
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      const int i = f.lane + 32 * s;
      if (i < n) X[i + size_t(j) * n] = i >= j ? start_f64(T[i + j * n] * f.rv[i]) : 0.0;
    }
  // the barriers' shared memory is used for other data next
  __syncthreads();
  if (int(threadIdx.x) < (n + 1) / 2) step_inval(&f.posted[threadIdx.x]);
}

// One 8 x 4 tile of a product: sum over k in [klo, khi) of A(i0 + i, k)
// B(k, j0 + j), element (r, k) of A at r ar + k ak, element (k, c) of B at
// c br + k bk (khi <= klo: no tile).
constexpr int kTileM = 8, kTileN = 4;
struct Tile {
  const double *A, *B;
  int ar, ak, br, bk, i0, j0, klo, khi;
};
constexpr int kBatch = 4;  // tiles a CTA stages at once: one load latency for all of them
constexpr int kTileElems = kTileM + 1 + kTileN + 1;  // staged doubles per k of a tile (odd strides)

// The CTA's tiles of one product phase: numbers first, first - stride, ... >=
// 0 (the long ones come last in every numbering, so they run first).  The
// operands of up to kBatch tiles are staged, warp w takes every eighth k of
// each, and warp q adds up tile q and hands output i = lane % 8, j = lane / 8
// to put(tile, row, column, value).  Operands may have been written by other
// CTAs before the last barrier: they are read through L2.
template <class Get, class Put>
__device__ void tile_products(int n, int first, int stride, Get get, Put put, double* sm) {
  constexpr int kLdA = kTileM + 1, kLdB = kTileN + 1, kWarps = kCoopThreads / 32;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  double* part = sm + size_t(kBatch) * n * kTileElems;  // kBatch x kCoopThreads
  for (int base = first; base >= 0; base -= kBatch * stride) {
    __syncthreads();  // the previous tiles' readers are done
#pragma unroll 1
    for (int q = 0; q < kBatch && base - q * stride >= 0; ++q) {
      const Tile f = get(base - q * stride);
      const int kt = f.khi - f.klo;
      double* sA = sm + size_t(q) * n * kTileElems;
      double* sB = sA + size_t(n) * kLdA;
#pragma unroll 4
      for (int idx = t; idx < kTileM * kt; idx += kCoopThreads) {
        const int r = f.ak == 1 ? idx / kt : idx % kTileM, k = f.ak == 1 ? idx - r * kt : idx / kTileM;
        sA[k * kLdA + r] = f.i0 + r < n ? __ldcg(&f.A[(f.i0 + r) * f.ar + (f.klo + k) * f.ak]) : 0.0;
      }
#pragma unroll 2
      for (int idx = t; idx < kTileN * kt; idx += kCoopThreads) {
        const int r = f.bk == 1 ? idx / kt : idx % kTileN, k = f.bk == 1 ? idx - r * kt : idx / kTileN;
        sB[k * kLdB + r] = f.j0 + r < n ? __ldcg(&f.B[(f.j0 + r) * f.br + (f.klo + k) * f.bk]) : 0.0;
      }
    }
    __syncthreads();
    const int i = lane & 7, j = lane >> 3;
#pragma unroll 1
    for (int q = 0; q < kBatch && base - q * stride >= 0; ++q) {
      const Tile f = get(base - q * stride);
      const int kt = f.khi - f.klo;
      const double* sA = sm + size_t(q) * n * kTileElems;
      const double* sB = sA + size_t(n) * kLdA;
      double acc = 0.0;
#pragma unroll 4
      for (int k = warp; k < kt; k += kWarps) acc = fma(sA[k * kLdA + i], sB[k * kLdB + j], acc);
      part[q * kCoopThreads + t] = acc;
    }
    __syncthreads();
    if (warp < kBatch && base - warp * stride >= 0) {
      const Tile f = get(base - warp * stride);
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += part[warp * kCoopThreads + 32 * w + lane];
      if (f.khi > f.klo && f.i0 + i < n && f.j0 + j < n) put(base - warp * stride, f.i0 + i, f.j0 + j, v);
    }
  }
}

// tile number -> (first row, first column) of the tiles that meet the lower
// triangle: row tile a has the column tiles 0 .. 2 a + 1
__device__ __forceinline__ void lower_tile(int tile, int& i0, int& j0) {
  static_assert(kTileM == 2 * kTileN, "two column tiles per row tile");
  int a = int((sqrtf(4.f * float(tile) + 1.f) - 1.f) * 0.5f);
  while (a * (a + 1) > tile) --a;
  while ((a + 1) * (a + 2) <= tile) ++a;
  i0 = a * kTileM;
  j0 = (tile - a * (a + 1)) * kTileN;
}

template <int SLOTS>
__global__ void __launch_bounds__(kCoopThreads, 1) thouless_evolve_kernel(EvolveArgs p) {
  extern __shared__ __align__(16) double evolve_smem[];
  const int n = p.n, t = threadIdx.x, G = gridDim.x, cta = blockIdx.x;
  unsigned gen = 0;  // barriers passed
  if (!p.newton) {
    evolve_by_blocks<SLOTS>(n, p.S, p.A, (long long)n * n, p.U1, p.V1 - p.U1, p.Linv, p.bar, gen, p.flags, p.skip_cta,
                            evolve_smem);
    return;
  }
  const size_t nn = size_t(n) * n;
  const int tm = (n + kTileM - 1) / kTileM, tn = (n + kTileN - 1) / kTileN;
  const int nlow = tm * (tm + 1);
  // S = 1 + Z^T Z, both triangles
  tile_products(
      n, nlow - 1 - cta, G,
      [&](int q) {
        Tile f{p.Z, p.Z, n, 1, n, 1, 0, 0, 0, n};
        lower_tile(q, f.i0, f.j0);
        if (f.j0 >= n) f.khi = 0;
        return f;
      },
      [&](int, int r, int c, double v) {
        if (c > r) return;
        const double s = r == c ? v + 1.0 : v;
        p.S[r + size_t(c) * n] = s;
        p.S[c + size_t(r) * n] = s;
      },
      evolve_smem);
  if (cta == p.skip_cta) return;  // test hook: the others' bounded waits run out
  if (!coop_barrier(p.bar, G, gen, p.flags)) return;
  // X0 by CTA 0; A1 = U0 + V0 Z and A2 = V0 + U0 Z by the others meanwhile
  const int per = tm * tn;
  if (cta == 0) {
    __syncthreads();
    if constexpr (SLOTS <= kF32MaxSlots) inverse_f32<SLOTS>(n, p.S, p.X0, evolve_smem, p.flags);
  }
  if (cta > 0 || G == 1)
    tile_products(
        n, 2 * per - 1 - (G > 1 ? cta - 1 : 0), G > 1 ? G - 1 : 1,
        [&](int q) {
          const int m = q / per, rest = q - m * per;
          return Tile{m ? p.U0 : p.V0, p.Z, 1, n, n, 1, rest % tm * kTileM, rest / tm * kTileN, 0, n};
        },
        [&](int q, int r, int c, double v) {
          const size_t at = r + size_t(c) * n;
          p.A[(q < per ? 0 : nn) + at] = v + __ldcg(&(q < per ? p.U0 : p.V0)[at]);
        },
        evolve_smem);
  if (!coop_barrier(p.bar, G, gen, p.flags)) return;
  double *X = p.X0, *Xn = p.X1;
  bool good = false;
  for (int step = 0; step < kNewtonSteps && !good; ++step) {
    // T = X S (the entries j <= i that the next product reads)
    tile_products(
        n, nlow - 1 - cta, G,
        [&](int q) {
          Tile f{X, p.S, 1, n, 1, n, 0, 0, 0, 0};
          lower_tile(q, f.i0, f.j0);
          f.khi = f.j0 < n ? min(f.i0 + kTileM, n) : 0;
          return f;
        },
        [&](int, int r, int c, double v) { p.T[r + size_t(c) * n] = v; }, evolve_smem);
    if (!coop_barrier(p.bar, G, gen, p.flags)) return;
    // E = Phi(T X^T - 1) and the largest entry of the residual
    float worst = 0.f;
    tile_products(
        n, nlow - 1 - cta, G,
        [&](int q) {
          Tile f{p.T, X, 1, n, 1, n, 0, 0, 0, 0};
          lower_tile(q, f.i0, f.j0);
          f.khi = f.j0 < n ? min(f.j0 + kTileN, n) : 0;
          return f;
        },
        [&](int, int r, int c, double v) {
          const double f = r == c ? v - 1.0 : v;
          p.E[r + size_t(c) * n] = c < r ? f : (c == r ? 0.5 * f : 0.0);
          if (c <= r) {
            const float m = fabsf(__double2float_rn(f));
            worst = m <= 1e30f ? fmaxf(worst, m) : 1e30f;  // NaN and infinity count as very large
          }
        },
        evolve_smem);
    for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if ((t & 31) == 0 && worst > 0.f) atomicMax(&p.bar[3 + step], __float_as_uint(worst));
    if (!coop_barrier(p.bar, G, gen, p.flags)) return;
    const float f = __uint_as_float(*(volatile unsigned*)&p.bar[3 + step]);
    if (!(f <= kNewtonUsable)) break;  // (uniform over the grid)
    good = f <= kNewtonLast;
    // X <- X - E X
    tile_products(
        n, nlow - 1 - cta, G,
        [&](int q) {
          Tile f{p.E, X, 1, n, n, 1, 0, 0, 0, 0};
          lower_tile(q, f.i0, f.j0);
          f.klo = f.j0;
          f.khi = min(f.i0 + kTileM, n);
          return f;
        },
        [&](int, int r, int c, double v) {
          const size_t at = r + size_t(c) * n;
          Xn[at] = c <= r ? __ldcg(&X[at]) - v : 0.0;
        },
        evolve_smem);
    if (!coop_barrier(p.bar, G, gen, p.flags)) return;
    double* swap = X;
    X = Xn;
    Xn = swap;
  }
  if (!good) {
    evolve_by_blocks<SLOTS>(n, p.S, p.A, (long long)nn, p.U1, p.V1 - p.U1, p.Linv, p.bar, gen, p.flags, -1,
                            evolve_smem);
    return;
  }
  // U1 = A1 X^T, V1 = A2 X^T
  tile_products(
      n, 2 * per - 1 - cta, G,
      [&](int q) {
        const int j0 = q / (2 * tm) * kTileN, rest = q % (2 * tm), m = rest / tm;
        return Tile{p.A + m * nn, X, 1, n, 1, n, rest % tm * kTileM, j0, 0, min(j0 + kTileN, n)};
      },
      [&](int q, int r, int c, double v) { (q % (2 * tm) < tm ? p.U1 : p.V1)[r + size_t(c) * n] = v; }, evolve_smem);
  if (p.Linv)
    for (size_t at = cta * size_t(kCoopThreads) + t; at < nn; at += size_t(G) * kCoopThreads)
      p.Linv[at] = at % n >= at / n ? __ldcg(&X[at]) : 0.0;
}

}  // namespace

size_t evolve_work(int n) { return size_t(7) * n * n + n; }

bool evolve_forms_products(int n) { return n <= kNewtonMaxN; }

int thouless_evolve(int n, const double* Z, const double* U0, const double* V0, double* work, double* U1, double* V1,
                    double* Linv, unsigned* bar, int* flags, cudaStream_t s, int skip_cta) {
  const size_t nn = size_t(n) * n;
  EvolveArgs p{};
  p.n = n;
  p.newton = evolve_forms_products(n) ? 1 : 0;
  p.Z = Z;
  p.U0 = U0;
  p.V0 = V0;
  p.A = work;
  p.S = work + 2 * nn;
  p.X0 = p.S + nn + n;
  p.X1 = p.X0 + nn;
  p.T = p.X1 + nn;
  p.E = p.T + nn;
  p.U1 = U1;
  p.V1 = V1;
  p.Linv = Linv;
  p.bar = bar;
  p.flags = flags;
  // shared memory: the FP32 stage's steps, the tiles' operands, the blocks'
  // panel rows
  size_t shm = sizeof(double) * (size_t(n) * kCoopNb + n);
  if (p.newton) {
    static_assert(kNewtonMaxN <= 32 * kF32MaxSlots, "the FP32 stage holds the matrix");
    shm = std::max(shm, sizeof(double) * n + sizeof(float) * (kF32Ring * (64 * kF32MaxSlots + 2) + n + 1 + nn));
    shm = std::max(shm, sizeof(double) * kBatch * (size_t(n) * kTileElems + kCoopThreads));
  }
  if (n > 384 || shm > jacobi32_smem_limit()) return TVAP_ERR_ARG;
  const int slots = (n + 31) / 32;
  const void* kern = slots <= 2    ? (const void*)thouless_evolve_kernel<2>
                     : slots <= 4  ? (const void*)thouless_evolve_kernel<4>
                     : slots <= 5  ? (const void*)thouless_evolve_kernel<5>
                     : slots <= 6  ? (const void*)thouless_evolve_kernel<6>
                     : slots <= 8  ? (const void*)thouless_evolve_kernel<8>
                     : slots <= 11 ? (const void*)thouless_evolve_kernel<11>
                                   : (const void*)thouless_evolve_kernel<12>;
  // the co-resident grid of this instantiation and shared-memory size, found
  // once per device
  struct GridKey {
    int dev;
    const void* kern;
    size_t shm;
  };
  static std::mutex m;
  static std::vector<std::pair<GridKey, int>> grids;
  int dev = 0;
  TVAP_CUDA(cudaGetDevice(&dev));
  int grid = 0;
  {
    std::lock_guard<std::mutex> lock(m);
    for (const auto& e : grids)
      if (e.first.dev == dev && e.first.kern == kern && e.first.shm == shm) grid = e.second;
    if (grid == 0) {
      if (int rc = smem_opt_in(kern, shm)) return rc;
      int per_sm = 0;
      TVAP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCoopThreads, shm));
      grid = std::min(per_sm * device_sms(), 128);
      if (grid >= 1) grids.push_back({GridKey{dev, kern, shm}, grid});
    }
  }
  if (grid < 1) return TVAP_ERR_ARG;
  TVAP_CUDA(cudaMemsetAsync(bar, 0, kEvolveBarWords * sizeof(unsigned), s));
  // small bases: no more CTAs than a product has tiles (a barrier of fewer CTAs is quicker)
  if (p.newton) grid = std::min(grid, std::max(2 * ((n + kTileM - 1) / kTileM) * ((n + kTileN - 1) / kTileN), 1));
  // the hook names the grid's last CTA (never CTA 0, which factors the
  // diagonal blocks); -1 leaves every CTA in
  p.skip_cta = (skip_cta >= 0 && grid > 1) ? grid - 1 : -1;
  void* args[] = {&p};
  ++g_launch_count;
  TVAP_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kCoopThreads), args,
                                        shm, s));
  return TVAP_OK;
}

}  // namespace tvap
