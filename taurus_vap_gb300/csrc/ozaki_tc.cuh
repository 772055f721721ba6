// The integer-splitting products of ozaki_core.cuh on the 5th-generation
// tensor cores (tcgen05): a warp-specialised pipeline fed by bulk asynchronous
// copies, accumulators in tensor memory, one thread issuing the MMAs.
//
// Digits.  Here an operand's integers |X| < 2^54 are written in balanced base
// 2^8: 7 digits of at most 128 (the leading one 64), all exact in bf16, and
// the 28 digit pairs (s, t) with s + t <= 6 are kept (the dropped ones sum to
// at most 6.03 * 2^54 units, what the 36 of 8 base-2^7 digits drop: 7.05).
// Seven planes instead of eight, 28 MMAs instead of 36.
//
// Every product reaching this path is a REAL product C' = A' B'^T of digit
// planes (complex operands are turned into real ones by the slicing pass).
// The slicing pass writes each digit plane already tiled in the tensor cores'
// canonical no-swizzle K-major layout, so that the operands of one k-step (16
// k, all 7 digits) of a 128-row A tile and of a 32-row B tile are contiguous
// blocks of 28 KB and 7 KB, fetched by one cp.async.bulk copy each.
//
// Tile layout (bf16 elements) of R rows x 16 k of one digit plane: R/8 row
// groups x 2 k-blocks of 8 x 8 "core matrices" (8 rows x 16 bytes, 128 bytes
// contiguous): element (r, k) at (r / 8) * 128 + (k / 8) * 64 + (r % 8) * 8 +
// k % 8.  Descriptor LBO = 128 B (next k-block), SBO = 256 B (next row group).
// The tiles of one operand are ordered [slot][row tile][k-step][digit].
//
// Persistent CTAs (one per SM) claim output tiles dynamically.  A CTA tile is
// 128 rows by one or two halves of 32 columns.  Each half has an accumulator
// set of its own in TMEM (7 weight groups g = s + t x 32 columns) and its own
// epilogue warps: warps 0-7 read set 0, warps 8-15 set 1 (warp w: TMEM lanes
// 32 (w % 4) .. + 32 = tile rows, columns 16 ((w / 4) % 2) .. + 16 of the
// half); warp 16 issues the copies, warp 17 the MMAs (issue_half: per half
// and k-step one MMA of N = 32 (7 - s) for each digit s of A).
//
// Over a fold interval of 160 k a group sum (at most 6 x 2^14 a k) stays below
// 2^24 and is an exact FP32 integer; at the end of an interval the epilogue
// warps read the set (tcgen05.ld) and fold it into 64-bit integer accumulators
// in registers.  While one set is read, the MMA warp runs the other half
// ahead by up to the stages of the pipeline, so the tensor pipe waits less for
// the folds (with one set of all 512 columns: 3400 cycles for each).  Measured
// cold against that form with 8 base-2^7 digits: H20's 280 x 560 x 140 for 113
// angles 215 -> 178 us, the solve's 280 x 56 x 252 112 -> 65 us, n = 336 672 x
// 1344 x 336 2023 -> 1464 us (1163 without the folds, 950 at the rate of the
// MMAs).
//
// Every wait is bounded: on a timeout the CTA raises its abort flag, stops
// issuing, waits (bounded) for the copies and MMAs it has issued and frees its
// tensor memory; the kernel then reports through the status word.
#pragma once

#include "ozaki_scaled.h"
#include "ozaki_core.cuh"

namespace tvap {
namespace oztc {

constexpr int kDigits = 7;
constexpr int kM = 128;                 // rows of A' per CTA tile (TMEM lanes)
constexpr int kHalf = 32;               // rows of B' (output columns) per half
constexpr int kSetWarps = 8;            // accumulator readers of a set
constexpr int kEpiWarps = 2 * kSetWarps;
constexpr int kProducerWarp = 16;       // bulk copies
constexpr int kMmaWarp = 17;            // TMEM allocation + MMA issue of set 0; 18: of set 1
constexpr int kThreads = 32 * (kEpiWarps + 3);
constexpr int kTmemCols = 512;
constexpr int kSetCols = 256;           // first column of set 1 (7 groups x 32 used of each)
constexpr int kStages = 5;
constexpr int kFoldKs = 10;             // k-steps per fold interval: 6 x 2^14 x 160 < 2^24
constexpr long long kSpin = 1LL << 21;  // bounded waits (polls)
// the product of two operands is (h 2^28 + l) 2^(ea + eb - kExpShift)
constexpr int kExpShift = 58;

constexpr int kATileElems = kM * 16;                // one digit plane of a k-step
constexpr int kBTileElems = kHalf * 16;
constexpr int kABytes = kDigits * kATileElems * 2;  // 28 KB per k-step
constexpr int kBBytes = kDigits * kBTileElems * 2;  // 7 KB per k-step and half
constexpr int kStageBytes = kABytes + 2 * kBBytes;
constexpr size_t kSmemBytes = size_t(kStages) * kStageBytes;
// one CTA per SM: two CTAs could never hold 512 TMEM columns each
static_assert(2 * kSmemBytes > 228 * 1024, "the tcgen05 kernel must not share an SM with itself");
static_assert(6LL * (1 << 14) * kFoldKs * 16 < (1 << 24), "group sums stay exact FP32 integers");

// balanced base-256 digits of |X| < 2^54, d[0] most significant: the low three
// from X mod 2^24 (leaving a carry of 0 or 1), the high four from the rest, in
// 32-bit arithmetic
__host__ __device__ __forceinline__ void to_digits(long long X, int* d) {
  int lo = int(X & 0xFFFFFFLL);
  int hi = int(X >> 24);
#pragma unroll
  for (int s = kDigits - 1; s >= 4; --s) {
    const int r = ((lo + 128) & 255) - 128;
    d[s] = r;
    lo = (lo - r) >> 8;
  }
  hi += lo;
#pragma unroll
  for (int s = 3; s >= 0; --s) {
    const int r = ((hi + 128) & 255) - 128;
    d[s] = r;
    hi = (hi - r) >> 8;
  }
}

#ifdef __CUDACC__
// bf16 bit patterns of the digits of two values (a in the low halves of w, b
// in the high ones) under the scale 2^emax, as to_digits(to_fixed()) gives
// them.  X + 128 (256^0 + .. + 256^6) is positive and its bytes are the
// balanced digits plus 128; a byte under the exponent of 2^23 minus 2^23 + 128
// is the digit as an FP32 number whose upper half is its bf16 pattern: three
// instructions a digit in place of seven.  The rounded shift has no branches:
// 2 mantissa >> t, half up, t = emax - exponent >= 0 (at most 63: nothing left).
__device__ __forceinline__ void digit_pair(double a, double b, int emax, uint32_t* w) {
  auto biased = [emax](double x) {
    const uint32_t hi = uint32_t(__double2hiint(x)), eb = (hi >> 20) & 0x7ffu;
    unsigned long long m = (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32) |
                           uint32_t(__double2loint(x));
    const int t = min(emax + 1023 - int(eb), 63);
    m = ((m << 1) + ((1ull << t) >> 1)) >> t;
    if (eb == 0) m = 0;  // zero and subnormal numbers
    constexpr unsigned long long kBias = 0x80808080808080ull;
    return int(hi) < 0 ? kBias - m : kBias + m;
  };
  const unsigned long long A = biased(a), B = biased(b);
#pragma unroll
  for (int s = 0; s < kDigits; ++s) {
    const int byte = kDigits - 1 - s;
    const uint32_t sel = 0x7540u + uint32_t(byte & 3);
    const uint32_t wa = byte < 4 ? uint32_t(A) : uint32_t(A >> 32), wb = byte < 4 ? uint32_t(B) : uint32_t(B >> 32);
    const float fa = __uint_as_float(__byte_perm(wa, 0x4B000000u, sel)) - 8388736.0f;
    const float fb = __uint_as_float(__byte_perm(wb, 0x4B000000u, sel)) - 8388736.0f;
    w[s] = __byte_perm(__float_as_uint(fa), __float_as_uint(fb), 0x7632);
  }
}
#endif

// element offset of (row r, k) inside the k-step tile of one digit plane
__host__ __device__ __forceinline__ int tile_offset(int r, int k) {
  return (r >> 3) * 128 + ((k >> 3) & 1) * 64 + (r & 7) * 8 + (k & 7);
}

#ifdef __CUDACC__

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t desc(uint32_t addr) {
  // start >> 4, LBO = 128 B, SBO = 256 B, descriptor version 1, no swizzle
  return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(128 >> 4) << 16) | (uint64_t(256 >> 4) << 32) |
         (uint64_t(1) << 46);
}

// kind::f16, bf16 x bf16 -> f32, both K-major, M = 128, N = n
__host__ __device__ constexpr uint32_t idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kM >> 4) << 24);
}

// Arrives when the MMAs that the elected thread of the (converged) warp issued
// before it are done.
__device__ __forceinline__ void commit(uint64_t* mbar) {
  asm volatile(
      "{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(mbar))
      : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(mbar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(smem_u32(mbar))
               : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(
                   smem_u32(mbar)),
               "r"(bytes)
               : "memory");
}

// bulk global -> shared copy completing `bytes` on an mbarrier (addresses
// 16-byte aligned, size a multiple of 16)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(mbar))
      : "memory");
}

__device__ __forceinline__ bool try_parity(uint64_t* mbar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(mbar)), "r"(parity)
      : "memory");
  return done != 0;
}

// bounded wait for the completion of phase `parity`; gives up early when the
// CTA's abort flag (if given) is raised.  `sleep` backs off between polls
// (for the many epilogue threads, so that they do not take issue slots from
// the producer and the MMA thread).
__device__ __forceinline__ bool wait_parity(uint64_t* mbar, uint32_t parity, volatile int* abort, bool sleep) {
  for (long long it = 0; it < kSpin; ++it) {
    if (try_parity(mbar, parity)) return true;
    if (abort && *abort) return false;
    if (sleep) __nanosleep(32);
  }
  return false;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// 8 consecutive 32-bit TMEM columns of the warp's 32 lanes
__device__ __forceinline__ void ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

// integer accumulators of one epilogue thread (16 columns): the product's
// integer is h 2^28 + l (groups 0 and 1 in h, 2-6 in l)
struct Acc {
  long long h[16], l[16];
};

constexpr int kRing = 4;  // tile numbers handed from the copy thread to the others

// shared control block
struct Ctl {
  uint64_t full[kStages], empty[kStages];
  uint64_t acc_full[2], acc_empty[2], mma_done[2];
  uint64_t tile_full[kRing], tile_empty[kRing];
  int tile_id[kRing];
  uint32_t tmem;
  int abort;
};

// MMAs of one half and k-step for all digit pairs (s, t), s + t <= 6.  The B
// digit tiles of a half lie back to back (digit t at + t KB, row groups 256 B
// apart), so digits 0 .. 6 - s form ONE K-major operand of 32 (7 - s) rows,
// whose accumulators (groups s .. 6) are adjacent TMEM column ranges: one MMA
// per digit s of A covers its 7 - s pairs.  FIRST = the k-step opens a fold
// interval: the products of s = 0, which reach every group, come first and
// overwrite the accumulators.  Otherwise the widest MMAs come last, so that
// the tensor pipe has work queued while the warp looks for the next k-step.
//
// Executed by the whole (converged) MMA warp, issued by its elected thread, in
// one statement: descriptors are read from uniform registers, which code that
// the compiler knows to be warp-uniform computes directly; in a branch of one
// thread every MMA first moved its six words from vector registers, about 110
// cycles an MMA, more than the MMA itself.
template <bool FIRST>
__device__ __forceinline__ void issue_half(uint32_t set, uint64_t da, uint64_t db) {
  static_assert(kDigits == 7 && kHalf == 32 && kATileElems == 2048, "the operands' steps below");
  if (FIRST) {
    asm volatile(
        "{\n.reg .pred q, z, o;\n.reg .b32 d1, d2, d3, d4, d5, d6;\n.reg .b64 a1, a2, a3, a4, a5, a6;\n"
        "setp.ne.u32 z, 0, 0;\nsetp.eq.u32 o, 0, 0;\n"
        "add.u32 d1, %0, 32;\nadd.u32 d2, %0, 64;\nadd.u32 d3, %0, 96;\nadd.u32 d4, %0, 128;\n"
        "add.u32 d5, %0, 160;\nadd.u32 d6, %0, 192;\n"
        "add.u64 a1, %1, 256;\nadd.u64 a2, %1, 512;\nadd.u64 a3, %1, 768;\nadd.u64 a4, %1, 1024;\n"
        "add.u64 a5, %1, 1280;\nadd.u64 a6, %1, 1536;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, z;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d6], a6, %2, %9, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d5], a5, %2, %8, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d4], a4, %2, %7, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d3], a3, %2, %6, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d2], a2, %2, %5, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d1], a1, %2, %4, o;\n}\n" ::"r"(set),
        "l"(da), "l"(db), "r"(idesc(224)), "r"(idesc(192)), "r"(idesc(160)), "r"(idesc(128)), "r"(idesc(96)),
        "r"(idesc(64)), "r"(idesc(32)));
  } else {
    asm volatile(
        "{\n.reg .pred q, o;\n.reg .b32 d1, d2, d3, d4, d5, d6;\n.reg .b64 a1, a2, a3, a4, a5, a6;\n"
        "setp.eq.u32 o, 0, 0;\n"
        "add.u32 d1, %0, 32;\nadd.u32 d2, %0, 64;\nadd.u32 d3, %0, 96;\nadd.u32 d4, %0, 128;\n"
        "add.u32 d5, %0, 160;\nadd.u32 d6, %0, 192;\n"
        "add.u64 a1, %1, 256;\nadd.u64 a2, %1, 512;\nadd.u64 a3, %1, 768;\nadd.u64 a4, %1, 1024;\n"
        "add.u64 a5, %1, 1280;\nadd.u64 a6, %1, 1536;\n"
        "elect.sync _|q, 0xffffffff;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d6], a6, %2, %9, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d5], a5, %2, %8, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d4], a4, %2, %7, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d3], a3, %2, %6, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d2], a2, %2, %5, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [d1], a1, %2, %4, o;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, o;\n}\n" ::"r"(set),
        "l"(da), "l"(db), "r"(idesc(224)), "r"(idesc(192)), "r"(idesc(160)), "r"(idesc(128)), "r"(idesc(96)),
        "r"(idesc(64)), "r"(idesc(32)));
  }
}

// Fold a set's group sums into the integer accumulators: h += S0 2^20 + S1 2^12,
// l += S2 2^32 + S3 2^24 + S4 2^16 + S5 2^8 + S6.  Neighbouring groups meet in
// 32 bits where they fit (|S0| < 2^20, |S1| < 2^22, |S2| < 2^23, |S3| < 2^23:
// S0 2^8 + S1 and S2 2^8 + S3), and the two smallest become integers by an
// FP32 addition (1.5 2^23 + S has S in its low bits for |S| <= 2^22), the
// others by conversions: 25 instructions a column for 42 with a 64-bit shift
// and add for each group (a set of 128 x 32: 2066 -> 1747 cycles by its 8 warps
// alone, 3791 -> 2856 for both sets at once).
// |l| grows by less than 2^55 a fold: 200 folds (kMaxKs) fit.
constexpr int kMaxKs = 2000;
__device__ __forceinline__ void fold(uint32_t set, Acc& o) {
  const int warp = threadIdx.x >> 5;
  const uint32_t at = set + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(((warp >> 2) & 1) * 16);
  constexpr uint32_t kMagic = 0x4B400000u;  // 1.5 2^23
  auto low = [](uint32_t u) { return __float_as_uint(__uint_as_float(u) + 12582912.0f); };
  auto num = [](uint32_t u) { return __float2int_rn(__uint_as_float(u)); };
#pragma unroll
  for (int c0 = 0; c0 < 16; c0 += 8) {
    uint32_t a[8], b[8];
    ld8(at + c0, a);
    ld8(at + kHalf + c0, b);
    ld_wait();
#pragma unroll
    for (int c = 0; c < 8; ++c) o.h[c0 + c] += (long long)int((low(a[c]) << 8) + low(b[c]) - kMagic * 257u) << 12;
    ld8(at + 2 * kHalf + c0, a);
    ld8(at + 3 * kHalf + c0, b);
    ld_wait();
#pragma unroll
    for (int c = 0; c < 8; ++c) o.l[c0 + c] += (long long)((num(a[c]) << 8) + num(b[c])) << 24;
    ld8(at + 4 * kHalf + c0, a);
    ld8(at + 5 * kHalf + c0, b);
    ld_wait();
#pragma unroll
    for (int c = 0; c < 8; ++c) o.l[c0 + c] += ((long long)num(a[c]) << 16) + ((long long)num(b[c]) << 8);
    ld8(at + 6 * kHalf + c0, a);
    ld_wait();
#pragma unroll
    for (int c = 0; c < 8; ++c) o.l[c0 + c] += (long long)num(a[c]);
  }
}

// Persistent driver, called by every thread of the CTA.  Tiles are claimed
// dynamically: the copy thread takes the next tile number from *counter
// (zero before the launch) and hands it to the MMA warp and the epilogue
// through a ring of kRing entries (mbarriers tile_full / tile_empty), so that
// CTAs that start late -- their SMs held by kernels of other streams -- take
// fewer tiles instead of delaying the product.  A number >= ntiles ends the
// CTA.  tile_ptrs(tile, A, B0, B1) gives the first k-step blocks of the tile's
// operands (nks_of(tile) k-steps of kABytes / kBBytes each follow
// contiguously), halves_of(tile) whether there is a second half (1 or 2);
// store(tile, half, acc) is called by the epilogue threads with their integer
// accumulators, after the set has been handed back to the MMA warp, so that
// the stores of one tile overlap the MMAs of the next.  The copy thread runs
// ahead across tile boundaries.  Returns false on a timeout.
template <class TilePtrs, class NksOf, class HalvesOf, class Store>
__device__ bool run_tiles(int* counter, int ntiles, NksOf nks_of, HalvesOf halves_of, unsigned char* smem, Ctl& ctl,
                          TilePtrs tile_ptrs, Store store) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort = &ctl.abort;
  if (threadIdx.x == 0) {
    for (int q = 0; q < kStages; ++q) {
      mbar_init(&ctl.full[q], 1);
      mbar_init(&ctl.empty[q], 2);
    }
    for (int q = 0; q < kRing; ++q) {
      mbar_init(&ctl.tile_full[q], 1);
      mbar_init(&ctl.tile_empty[q], kEpiWarps + 2);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(&ctl.acc_full[q], 1);
      mbar_init(&ctl.acc_empty[q], kSetWarps);
      mbar_init(&ctl.mma_done[q], 1);
    }
    ctl.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&ctl.tmem)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = ctl.tmem;
  bool ok = true;
  uint32_t issued = 0;  // k-steps whose copies were issued (copy thread)
  if (warp == kProducerWarp) {
    if (lane == 0) {
      int st = 0;           // stage
      uint32_t par = 1;     // parity of the phase before the stage's next one
      for (int tt = 0; ok; ++tt) {
        const int slot = tt % kRing;
        if (tt >= kRing && !wait_parity(&ctl.tile_empty[slot], uint32_t((tt / kRing - 1) & 1), abort, false)) {
          ok = false;
          break;
        }
        int tile = atomicAdd(counter, 1);
        if (tile >= ntiles) tile = -1;
        ctl.tile_id[slot] = tile;
        mbar_arrive(&ctl.tile_full[slot]);
        if (tile < 0) break;
        const unsigned char *A, *B0, *B1;
        tile_ptrs(tile, A, B0, B1);
        const int nks = nks_of(tile);
        const bool two = halves_of(tile) > 1;
        for (int ks = 0; ks < nks; ++ks) {
          if (issued >= uint32_t(kStages) && !wait_parity(&ctl.empty[st], par, abort, false)) {
            ok = false;
            break;
          }
          unsigned char* dst = smem + st * kStageBytes;
          mbar_expect_tx(&ctl.full[st], uint32_t(kABytes + (two ? 2 : 1) * kBBytes));
          bulk_load(dst, A, uint32_t(kABytes), &ctl.full[st]);
          bulk_load(dst + kABytes, B0, uint32_t(kBBytes), &ctl.full[st]);
          if (two) bulk_load(dst + kABytes + kBBytes, B1, uint32_t(kBBytes), &ctl.full[st]);
          A += kABytes;
          B0 += kBBytes;
          B1 += kBBytes;
          ++issued;
          if (++st == kStages) {
            st = 0;
            par ^= 1;
          }
        }
      }
    }
  } else if (warp >= kMmaWarp) {
    // One warp per set, each at its own pace: a half-tile's k-step costs a warp
    // about 700 cycles (waits, seven MMAs, commits), the tensor pipe 480.  A
    // stage is free when both are done with it.  The whole warp runs this
    // loop, converged (mma()); what it reads from shared memory is broadcast,
    // so that the compiler knows it to be uniform.
    const int s = warp - kMmaWarp;
    const uint32_t set = __shfl_sync(0xffffffffu, tmem, 0) + uint32_t(s * kSetCols);
    const uint64_t base = desc(smem_u32(smem));
    int st = 0;              // stage
    uint32_t par = 0;        // and the parity of its phase
    uint32_t fc = 0;         // fold intervals over all tiles
    auto wait = [&](uint64_t* mbar, uint32_t parity) {
      return __all_sync(0xffffffffu, wait_parity(mbar, parity, abort, false)) != 0;
    };
    for (int tt = 0; ok; ++tt) {
      const int slot = tt % kRing;
      if (!wait(&ctl.tile_full[slot], uint32_t((tt / kRing) & 1))) {
        ok = false;
        break;
      }
      const int tile = __shfl_sync(0xffffffffu, ctl.tile_id[slot], 0);
      if (lane == 0) mbar_arrive(&ctl.tile_empty[slot]);
      __syncwarp();
      if (tile < 0) break;
      const int nks = __shfl_sync(0xffffffffu, nks_of(tile), 0);
      const bool mine = __shfl_sync(0xffffffffu, halves_of(tile), 0) > s;
      int left = 0;  // k-steps left in the fold interval
      for (int ks = 0; ks < nks; ++ks) {
        // a new interval overwrites the accumulators: the epilogue must have
        // read the previous one
        if (!wait(&ctl.full[st], par) || (mine && left == 0 && fc > 0 && !wait(&ctl.acc_empty[s], (fc - 1) & 1))) {
          ok = false;
          break;
        }
        if (mine) {
          fence_after();
          const uint64_t da = base + uint64_t(st * (kStageBytes >> 4));
          const uint64_t db = da + uint64_t((kABytes + s * kBBytes) >> 4);
          if (left == 0) {
            issue_half<true>(set, da, db);
            left = min(kFoldKs, nks - ks);
          } else {
            issue_half<false>(set, da, db);
          }
          commit(&ctl.empty[st]);
          if (--left == 0) {
            commit(&ctl.acc_full[s]);
            ++fc;
          }
        } else if (lane == 0) {
          mbar_arrive(&ctl.empty[st]);
        }
        if (++st == kStages) {
          st = 0;
          par ^= 1;
        }
      }
    }
    // every MMA issued by this warp has completed once its mma_done flips
    commit(&ctl.mma_done[s]);
    wait_parity(&ctl.mma_done[s], 0u, nullptr, false);
    __syncwarp();
  } else {
    // the epilogue warps decide as whole warps (a lane that gives up takes its
    // warp with it): the accumulator loads are warp-wide (.sync.aligned) and
    // the paired store shuffles between lanes
    const int s = warp / kSetWarps;
    uint32_t fc = 0;
    // one arrival per warp (the arrivals of all its threads on one barrier run
    // one after the other in shared memory)
    auto warp_arrive = [&](uint64_t* mbar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(mbar);
    };
    for (int tt = 0; ok; ++tt) {
      const int slot = tt % kRing;
      if (!__all_sync(0xffffffffu, wait_parity(&ctl.tile_full[slot], uint32_t((tt / kRing) & 1), abort, true))) {
        ok = false;
        break;
      }
      const int tile = ctl.tile_id[slot];
      warp_arrive(&ctl.tile_empty[slot]);
      if (tile < 0) break;
      if (s >= halves_of(tile)) continue;
      const int nfold = (nks_of(tile) + kFoldKs - 1) / kFoldKs;  // fold intervals of the tile
      Acc o;
#pragma unroll
      for (int c = 0; c < 16; ++c) o.h[c] = o.l[c] = 0;
      for (int f = 0; f < nfold; ++f, ++fc) {
        if (!__all_sync(0xffffffffu, wait_parity(&ctl.acc_full[s], fc & 1, abort, true))) {
          ok = false;
          break;
        }
        fence_after();
        fold(tmem + uint32_t(s * kSetCols), o);
        fence_before();
        warp_arrive(&ctl.acc_empty[s]);
      }
      if (ok) store(tile, s, o);
    }
  }
  if (!ok) ctl.abort = 1;
  fence_before();
  __syncthreads();
  const bool all_ok = ctl.abort == 0;
  if (!all_ok && warp == kProducerWarp && lane == 0) {
    // the copies in flight land before the shared memory is released: the
    // last phase of each stage's barrier is that of its last copy
    for (uint32_t it = (issued > kStages ? issued - kStages : 0); it < issued; ++it)
      wait_parity(&ctl.full[it % kStages], (it / kStages) & 1, nullptr, false);
  }
  if (warp == kMmaWarp) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTmemCols));
  }
  return all_ok;
}

// value of column c (0..15 of the thread's quarter) before the exponent scale
__device__ __forceinline__ double value(const Acc& o, int c) { return fma(double(o.h[c]), 0x1p28, double(o.l[c])); }


#endif  // __CUDACC__

}  // namespace oztc
}  // namespace tvap
