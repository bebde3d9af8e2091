// FP64-accurate correlation Gram on the 5th-generation tensor cores (tcgen05 + TMA),
// by exact integer digits (an Ozaki-style splitting).
//
// Replaces the reference's FP64 gpuPMCC (src/correlation/corHelper.cu:79-116) where
// the correlation has to be FP64-accurate (HPC_PREC_MIXED): GB300's FP64 pipe gives
// about 1 TFLOP/s, so the p=2000, n=5000 Gram takes 20 ms in SIMT FP64; here it runs
// as BF16 tensor-core products that are exact.
//
//   y_v = z_v * 2^-e_v                  (e_v: the exponent of max |z_v|, so |y_v| <= 1)
//   y_v = sum_{t=1..7} d_t(v) 2^-7t     (d_1 = rint(128 y), then the remainders 7 bits
//                                        at a time: integers, |d_1| <= 128, |d_t| <= 64,
//                                        all exact in BF16; 49 bits of y)
//   sum_k y_a y_b = sum_{t+u<=8} 2^-7(t+u) sum_k d_t(a) d_u(b)   (weights below 2^-56 dropped)
//
// Each digit product is an integer of at most 2^14, so sums of a few hundred samples over
// all the pairs (t, u) of one weight s = t + u are integers of at most 2^24: exact in the
// tensor core's FP32 accumulator. The kernel keeps one TMEM accumulator per weight and runs
// a block of 32 samples' digits against each other while they stand in shared memory: 56
// MMAs for 112 KB of operands, where a pair at a time needs 28 times 16 KB. Seven 128-column
// accumulators exceed the 512 columns of TMEM, so the samples go by twice: first the weights 6..8
// (all digits: 18 pairs), then 2..5 (digits 1..4: 10 pairs). Every kGroupStages stages the
// drain warps add the exact sums into 64-bit fixed-point integers with integer instructions --
// the FP64 pipe would be the bottleneck -- one weight after the other, while the MMAs of the
// others go on. The first pass's integers have an LSB of 2^-56 of sum y_a y_b, which every weight
// is a multiple of; between the passes they become an LSB of 2^-47 (the range of the whole sum for
// n <= 32768) and the kLowBits below it. Where there are fewer tiles than SMs a cluster of blocks
// shares a tile's samples; it adds up both through distributed shared memory and rounds once, as
// a block alone does: the result does not depend on the split. The epilogue scales by
// 2^(e_a + e_b) / (n - 1) and writes the FP64 entry (both triangles) and its FP32 rounding.
//
// Error of an entry, beside the roundings of FP64: the digits' 49 bits, at most 2^-50 (2^e_a +
// 2^e_b); the dropped pairs, at most 6 * 2^12 * 2^-63 (1 + 2^-6) a sample, 2^(e_a + e_b - 48.3); the
// rounding, 2^(e_a + e_b - 48) / (n - 1). 2^e is 8 for Gaussian data and at most 2 sqrt(n - 1), where one
// sample outweighs all others. The dropped pairs' signs vary, so that they add up to far less:
// measured against 113 bits, p = 257..2000, n = 2000..32768, the largest error is 1.2e-15 on Gaussian
// data and 3.8e-13 where one sample of each variable is a thousand times the others (2.6e-15 and
// 1.4e-12 with every group's sums of the weights 7 and 8 rounded down to 2^-47).
//
// Structure (one CTA of 10 warps per tile and part): warp 0 lane 0 TMA producer, warp 1 lane 0
// MMA issuer (tcgen05.mma.kind::f16, M = N = 128, K = 16), warps 2-9 drain (TMEM lane quadrant
// warp % 4, 64 columns each). Every mbarrier wait is bounded; on time-out the CTA records
// kErrTimeout, stops issuing, waits (bounded) for its copies and MMAs, frees its TMEM and
// returns.
//
// Bound: the tensor cores and, beside them, the shared memory they read the operands from
// (64 of every 80 cycles). Measured (this kernel): p = 2000, n = 5000 918 us with a pair at a
// time, 462 us now (6.4e11 flops: 1.4 PFLOP/s; 497 us with a drain that shifts both ways, which the
// first pass's LSB saves); p = 1203, n = 3777, on 55 of 152 SMs then, 746 -> 193 us. The digits
// 616 -> 53 us and 317 -> 27 us.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.cuh"
#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace hpc {
namespace {

constexpr int EM = 128, EN = 128, EK = 32;   // tile 128 x 128, 32 samples (64 B of a digit) per stage
constexpr int kDigits = 7;
constexpr int kTileBytes = EM * EK * 2;      // one digit's 128 rows of a stage: 8 KB
// The two passes: weights s = 6..8 and 2..5 (accumulators 0..2 and 0..3), the digits they
// need, and their stages -- both cut the same 224 KB, of which the second leaves 32 KB: there a
// block of a cluster keeps its sums' low bits meanwhile.
constexpr int kDigitsA = 7, kSlotsA = 3, kStagesA = 2, kBytesA = 2 * kDigitsA * kTileBytes;
constexpr int kDigitsB = 4, kSlotsB = 4, kStagesB = 3, kBytesB = 2 * kDigitsB * kTileBytes;
constexpr int kFirstA = 6, kFirstB = 2;  // their lowest weights
constexpr int kOperandBytes = kStagesA * kBytesA;
// Stages between two drains: the largest weight's sum grows by (2 * 2^13 + 5 * 2^12) a sample at
// most (d_1 against d_7 twice, |d_1| <= 128, and five pairs of |d| <= 64), so 448 samples
// stay below 2^24
constexpr int kGroupStages = 14;
static_assert((2 * 8192 + 5 * 4096) * kGroupStages * EK <= (1 << 24), "exact in FP32");
constexpr int kTmemColsE = 512;              // four 128-column accumulators
constexpr int kAccWarpsE = 8;
constexpr int kThreadsE = 64 + 32 * kAccWarpsE;
constexpr int kFixL = 47;                    // fixed-point LSB 2^-47
constexpr int kLowBits = 9;                  // ... and the first pass's 2^-56
constexpr int kMaxSplitE = 8;                // portable cluster size

struct alignas(1024) EmuSmem {
  uint8_t operands[kOperandBytes];  // the stages; at the end a block's 128 x 128 integer sums
  uint64_t full_a[kStagesA], empty_a[kStagesA];
  uint64_t full_b[kStagesB], empty_b[kStagesB];
  uint64_t acc_full[kSlotsB], acc_empty[kSlotsB];
  uint64_t drain;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(EmuSmem) + 1024 <= 227 * 1024, "shared memory of a block");
constexpr int kLowAt = kStagesB * kBytesB;   // the low bits, [column][row]
static_assert(kLowAt + sizeof(uint16_t) * EM * EN <= kOperandBytes, "beside the second pass's stages");
static_assert(sizeof(long long) * EM * EN <= kLowAt, "the sums fit before them");
static_assert(kFixL + kLowBits == 7 * 8, "no bit of the lowest weight is lost");

__device__ __forceinline__ bool aborted(EmuSmem &sm) { return *(volatile int *)&sm.abort != 0; }
__device__ __forceinline__ void fail(EmuSmem &sm, int *err) {
  atomicOr(err, kErrTimeout);
  atomicExch(&sm.abort, 1);
}

// One block per variable (rows beyond p are written as zero digits): the exponent of max |z|
// and the seven digits of z * 2^-e for every sample (zero beyond n, and for a sample that is
// not finite). All in integers on the bits of z -- rounded to 49 bits, then cut 7 bits at a
// time -- since the FP64 pipe (2 results a clock and SM) took 616 us for p = 2000, n = 5000 where
// the 220 MB of traffic take 32. Four samples a thread, so that a digit's four go out as 8 bytes.
__global__ void __launch_bounds__(256) emu_digits_kernel(const double *__restrict__ Z, int64_t p, int64_t n,
                                                         int64_t n_pad, __nv_bfloat16 *__restrict__ D,
                                                         int *__restrict__ E) {
  const int64_t v = blockIdx.x;
  __nv_bfloat16 *dv = D + v * (int64_t)kDigits * n_pad;
  const long long *zv = reinterpret_cast<const long long *>(Z + v * n);
  __shared__ int red[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int ex = 0;  // largest biased exponent of a finite sample (0: all zero or denormal)
  if (v < p)
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) {
      const int x = (int)(__ldg(zv + k) >> 52) & 0x7ff;
      if (x < 0x7ff) ex = max(ex, x);
    }
  ex = __reduce_max_sync(0xffffffffu, ex);
  if (lane == 0) red[wid] = ex;
  __syncthreads();
  int e = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, red[w]);
  e = e ? e - 1022 : 0;  // max |z| = f 2^e, f in [0.5, 1)
  if (threadIdx.x == 0) E[v] = e;
  for (int64_t k = 4 * (int64_t)threadIdx.x; k < n_pad; k += 4 * blockDim.x) {
    uint32_t dig[kDigits][4];  // FP32 bits of the digits: small integers, exact in their upper half
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long bits = v < p && k + u < n ? __ldg(zv + k + u) : 0ll;
      const int x = (int)(bits >> 52) & 0x7ff;
      // N = rint(|z| 2^(49 - e)): the 53-bit mantissa shifted right by sh >= 4, to nearest even
      const int sh = 1026 + e - x;
      const unsigned long long m = ((unsigned long long)bits & 0xfffffffffffffull) | (1ull << 52);
      long long N = 0;
      if (x != 0 && x != 0x7ff && sh < 60)
        N = (long long)((m + ((1ull << (sh - 1)) - 1ull) + ((m >> sh) & 1ull)) >> sh);
      if (bits < 0) N = -N;
      // digits 7..5 in 64 bits, the other 28 bits in 32
#pragma unroll
      for (int t = kDigits - 1; t >= 4; --t) {
        const int d = ((int)(N + 64) & 127) - 64;
        N = (N - d) >> 7;
        dig[t][u] = __float_as_uint((float)d);
      }
      int M = (int)N;
#pragma unroll
      for (int t = 3; t >= 1; --t) {
        const int d = ((M + 64) & 127) - 64;
        M = (M - d) >> 7;
        dig[t][u] = __float_as_uint((float)d);
      }
      dig[0][u] = __float_as_uint((float)M);
    }
#pragma unroll
    for (int t = 0; t < kDigits; ++t)
      *reinterpret_cast<uint2 *>(dv + t * n_pad + k) =
          make_uint2(__byte_perm(dig[t][0], dig[t][1], 0x7632), __byte_perm(dig[t][2], dig[t][3], 0x7632));
  }
}

__global__ void __launch_bounds__(kThreadsE, 1)
    gram_emu_kernel(const __grid_constant__ CUtensorMap map, int64_t p, int64_t n_pad, double denom,
                    const int *__restrict__ E, double *__restrict__ C64, float *__restrict__ C32, int *err, int split) {
  extern __shared__ uint8_t smem_raw[];
  EmuSmem &sm = *reinterpret_cast<EmuSmem *>((((uintptr_t)smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // tile (bi, bj), bi <= bj, row-major over the upper triangle of 128-blocks, and the block's part
  // of the samples
  const int nb = (int)((p + EM - 1) / EM);
  const int part = (int)(blockIdx.x % (unsigned)split);
  long long t = blockIdx.x / (unsigned)split;
  int bi = 0;
  while (t >= nb - bi) {
    t -= nb - bi;
    ++bi;
  }
  const int bj = bi + (int)t;
  const int stages = (int)(n_pad / EK);
  const int kb0 = (int)((long long)stages * part / split), kb1 = (int)((long long)stages * (part + 1) / split);
  const int nk = kb1 - kb0;
  const int groups = (nk + kGroupStages - 1) / kGroupStages;
  const uint32_t idesc = idesc_bf16(EM, EN);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesA; ++s) {
      mbar_init(&sm.full_a[s], 1);
      mbar_init(&sm.empty_a[s], 1);
    }
    for (int s = 0; s < kStagesB; ++s) {
      mbar_init(&sm.full_b[s], 1);
      mbar_init(&sm.empty_b[s], 1);
    }
    for (int c = 0; c < kSlotsB; ++c) {
      mbar_init(&sm.acc_full[c], 1);
      mbar_init(&sm.acc_empty[c], kAccWarpsE);
    }
    mbar_init(&sm.drain, 1);
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(kTmemColsE));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sm.tmem_base;

  int issued_a = 0, issued_b = 0;
  constexpr int kCols = EN / 2;
  long long acc[kCols];  // drain warps: the thread's row, 64 columns
  bool ok = true;
  if (warp == 0 && lane == 0) {
    // TMA producer: each stage's digits of the rows (block bi) and of the columns (block bj)
    auto load = [&](uint8_t *to, int digits, int kb, uint64_t *bar) {
      for (int d = 0; d < digits; ++d) {
        tma_load_2d(to + d * kTileBytes, &map, (int)(d * n_pad) + kb * EK, bi * EM, bar);
        tma_load_2d(to + (digits + d) * kTileBytes, &map, (int)(d * n_pad) + kb * EK, bj * EN, bar);
      }
    };
    for (int k = 0; k < nk; ++k) {
      const int s = k % kStagesA;
      if (k >= kStagesA && !mbar_wait(&sm.empty_a[s], ((k / kStagesA) + 1) & 1)) {
        fail(sm, err);
        break;
      }
      if (aborted(sm)) break;
      mbar_arrive_expect_tx(&sm.full_a[s], kBytesA);
      load(sm.operands + s * kBytesA, kDigitsA, kb0 + k, &sm.full_a[s]);
      ++issued_a;
    }
    // the second pass overwrites the first one's stages: all of them have been read
    for (int s = 0; s < kStagesA && !aborted(sm); ++s) {
      const int fills = issued_a / kStagesA + (s < issued_a % kStagesA ? 1 : 0);
      if (fills > 0 && !mbar_wait(&sm.empty_a[s], (fills - 1) & 1)) fail(sm, err);
    }
    for (int k = 0; k < nk && !aborted(sm); ++k) {
      const int s = k % kStagesB;
      if (k >= kStagesB && !mbar_wait(&sm.empty_b[s], ((k / kStagesB) + 1) & 1)) {
        fail(sm, err);
        break;
      }
      if (aborted(sm)) break;
      mbar_arrive_expect_tx(&sm.full_b[s], kBytesB);
      load(sm.operands + s * kBytesB, kDigitsB, kb0 + k, &sm.full_b[s]);
      ++issued_b;
    }
  } else if (warp == 1 && lane == 0) {
    // MMA issuer. Pass P: accumulator c takes the digit pairs of weight first + c; a stage's MMAs of
    // one accumulator after the other, so that a drained one is refilled while the next is drained.
    // fill: how often the first kSlotsA accumulators were filled before (their barriers' phases)
    auto run = [&](int first, int slots, int digits, int nstages, int bytes, uint64_t *full, uint64_t *empty,
                   int fill) {
      for (int k = 0; k < nk && !aborted(sm); ++k) {
        const int s = k % nstages, g = k / kGroupStages;
        const bool begin = k % kGroupStages == 0, end = k == nk - 1 || (k + 1) % kGroupStages == 0;
        if (!mbar_wait(&full[s], (k / nstages) & 1)) {
          fail(sm, err);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_u32(sm.operands + s * bytes), b0 = a0 + digits * kTileBytes;
        for (int c = 0; c < slots; ++c) {
          const int before = (c < kSlotsA ? fill : 0) + g;
          if (begin && before > 0) {
            if (!mbar_wait(&sm.acc_empty[c], (before - 1) & 1)) {
              fail(sm, err);
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          }
          const int sum = first - 2 + c;  // 0-based digits t + u
          for (int t0 = 0; t0 <= sum; ++t0) {
            const uint32_t a = a0 + t0 * kTileBytes, bb = b0 + (sum - t0) * kTileBytes;
#pragma unroll
            for (int kk = 0; kk < EK / 16; ++kk)
              mma_bf16(tmem + (uint32_t)(c * EN), smem_desc_sw64(a + kk * 32), smem_desc_sw64(bb + kk * 32), idesc,
                       (begin && t0 == 0 && kk == 0) ? 0u : 1u);
          }
          if (end) mma_commit(&sm.acc_full[c]);
        }
        mma_commit(&empty[s]);
      }
    };
    run(kFirstA, kSlotsA, kDigitsA, kStagesA, kBytesA, sm.full_a, sm.empty_a, 0);
    run(kFirstB, kSlotsB, kDigitsB, kStagesB, kBytesB, sm.full_b, sm.empty_b, groups);
    mma_commit(&sm.drain);
    if (!mbar_wait(&sm.drain, 0)) fail(sm, err);
  } else if (warp >= 2) {
    // drain: rows 32 (warp % 4) .. + 31 (TMEM lanes), columns 64 ((warp - 2) / 4) .. + 63
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
#pragma unroll
    for (int q = 0; q < kCols; ++q) acc[q] = 0;
    for (int pass = 0; pass < 2 && ok; ++pass) {
      const int slots = pass ? kSlotsB : kSlotsA, first = pass ? kFirstB : kFirstA;
      const int lsb = pass ? kFixL : kFixL + kLowBits;
      for (int g = 0; g < groups && ok; ++g)
        for (int c = 0; c < slots; ++c) {
          if (!mbar_wait(&sm.acc_full[c], ((pass && c < kSlotsA ? groups : 0) + g) & 1)) {
            fail(sm, err);
            ok = false;
            break;
          }
          __syncwarp();
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int sh = lsb - 7 * (first + c);  // the sum's weight 2^-7s in units of 2^-lsb
#pragma unroll
          for (int c0 = 0; c0 < kCols; c0 += 16) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c * EN + half * kCols + c0), v);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const long long gi = (long long)__float2int_rn(v[q]);  // an integer of at most 2^24: exact
              acc[c0 + q] += (long long)((unsigned long long)gi << sh);
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.acc_empty[c]);
        }
      if (pass == 0 && ok) {
        // to the LSB of the whole sum: rounded, or with the low bits kept for the cluster's sum (the first
        // pass's MMAs have all completed, and the second's copies end before kLowAt)
        uint16_t *low = reinterpret_cast<uint16_t *>(sm.operands + kLowAt) + half * kCols * EM + quad * 32 + lane;
#pragma unroll
        for (int q = 0; q < kCols; ++q) {
          if (split > 1) low[q * EM] = (uint16_t)(acc[q] & ((1 << kLowBits) - 1));
          else acc[q] += 1 << (kLowBits - 1);
          acc[q] >>= kLowBits;
        }
      }
    }
  }
  __syncwarp();
  // one entry: scaled, both triangles. 1 / denom times a power of two: one multiplication (a
  // division's FP64 instructions would take 40 us at p = 2000)
  const double inv = 1.0 / denom;
  auto write = [&](int64_t row, int64_t col, long long sum, int er) {
    if (row < p && col < p && col >= row) {
      const double scale = __hiloint2double(__double2hiint(inv) + ((er + E[col] - kFixL) << 20), __double2loint(inv));
      const double v = (double)sum * scale;
      C64[col * p + row] = v;  // the warp's lanes: consecutive rows, one column
      C64[row * p + col] = v;
      if (C32) {
        C32[col * p + row] = (float)v;
        C32[row * p + col] = (float)v;
      }
    }
  };
  const int64_t row = (int64_t)bi * EM + (warp & 3) * 32 + lane;
  const int er = warp >= 2 && row < p ? E[row] : 0;
  if (split == 1) {
    if (warp >= 2 && ok && !aborted(sm)) {
      const int64_t col0 = (int64_t)bj * EN + ((warp - 2) >> 2) * kCols;
#pragma unroll
      for (int cc = 0; cc < kCols; ++cc) write(row, col0 + cc, acc[cc], er);
    }
  } else {
    // the parts' sums: each block keeps its own in its operand buffer (every copy and MMA has
    // completed; the low bits stand behind), then adds up and writes its share of the columns
    cg::cluster_group cluster = cg::this_cluster();
    long long *sums = reinterpret_cast<long long *>(sm.operands);  // [column][row]
    __syncthreads();
    if (warp >= 2) {
      const int c0 = ((warp - 2) >> 2) * kCols, r = (warp & 3) * 32 + lane;
#pragma unroll
      for (int cc = 0; cc < kCols; ++cc) sums[(c0 + cc) * EM + r] = acc[cc];
    }
    cluster.sync();
    if (warp >= 2 && !aborted(sm)) {  // a part that failed has raised err: the host does not use C
      const int r = (warp & 3) * 32 + lane;
      const int lo = EN * part / split, hi = EN * (part + 1) / split;
      for (int cc = lo + ((warp - 2) >> 2); cc < hi; cc += 2) {
        long long sum = 0;
        int low = 1 << (kLowBits - 1);
        for (int q = 0; q < split; ++q) {
          sum += cluster.map_shared_rank(sums, q)[cc * EM + r];
          low += cluster.map_shared_rank(reinterpret_cast<uint16_t *>(sm.operands + kLowAt), q)[cc * EM + r];
        }
        write(row, (int64_t)bj * EN + cc, sum + (low >> kLowBits), er);
      }
    }
    cluster.sync();  // no block leaves while its sums are read
  }
  if (warp == 0 && lane == 0 && sm.abort) {
    for (int s = 0; s < kStagesA; ++s) {
      const int fills = issued_a / kStagesA + (s < issued_a % kStagesA ? 1 : 0);
      if (fills > 0) mbar_wait(&sm.full_a[s], (fills - 1) & 1);
    }
    for (int s = 0; s < kStagesB; ++s) {
      const int fills = issued_b / kStagesB + (s < issued_b % kStagesB ? 1 : 0);
      if (fills > 0) mbar_wait(&sm.full_b[s], (fills - 1) & 1);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColsE));
  }
}

int64_t emu_n_pad(int64_t n) { return (n + EK - 1) / EK * EK; }

// Blocks a tile's samples are split over: the largest power of two (up to a portable cluster)
// with which every block still runs at once, one an SM, and keeps a group of stages or more.
// (Of clusters of 2, 4 and 8 the GPU holds 76, 36 and 15 at once; the rule's largest triangles of
// tiles are 66, 36 and 15.)
int emu_split(long long tiles, int64_t n_pad) {
  int split = 1;
  while (split < kMaxSplitE && tiles * split * 2 <= 152 && n_pad / (split * 2) >= kGroupStages * EK) split *= 2;
  return split;
}

}  // namespace

// The exact-digit Gram serves one instance of at least 256 variables (below that the
// SIMT FP64 Gram is as fast) and at most 32768 samples (the fixed point's range).
bool emu_eligible(int64_t p, int64_t n) { return p >= 256 && n <= 32768; }
int64_t emu_p_pad(int64_t p) { return (p + EM - 1) / EM * EM; }
int64_t emu_digit_elems(int64_t p, int64_t n) { return emu_p_pad(p) * kDigits * emu_n_pad(n); }

hpc_status launch_gram_emu(const double *Z, int64_t p, int64_t n, double denom, __nv_bfloat16 *D, int *E,
                           CUtensorMap * /*unused*/, double *C64, float *C32, int *err, cudaStream_t s) {
  const int64_t n_pad = emu_n_pad(n), p_pad = emu_p_pad(p);
  emu_digits_kernel<<<(unsigned)p_pad, 256, 0, s>>>(Z, p, n, n_pad, D, E);
  HPC_LAUNCH_CHECK("emu_digits_kernel");
  CUtensorMap map;
  hpc_status st = tc_make_map(&map, D, p_pad, kDigits * n_pad, EM, EK);
  if (st != HPC_OK) return st;
  const int smem = (int)sizeof(EmuSmem) + 1024;
  HPC_CUDA(cudaFuncSetAttribute(gram_emu_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const long long nb = p_pad / EM, tiles = nb * (nb + 1) / 2;
  const int split = emu_split(tiles, n_pad);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * split));
  cfg.blockDim = dim3(kThreadsE);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HPC_CUDA(cudaLaunchKernelEx(&cfg, gram_emu_kernel, map, p, n_pad, denom, (const int *)E, C64, C32, err, split));
  return HPC_OK;
}

}  // namespace hpc
