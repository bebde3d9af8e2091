// Correlation: column standardisation and the FP64 Gram, grouped over the instances
// of a context.
//
// Replaces gpuMeans / gpuSD / gpuPMCC (src/correlation/corHelper.cu:8-116), which
// launch one 64-thread block per (i, j) pair and re-read both columns for every pair.
// Here one block per variable standardises its column once (NaN-skipping mean, SD with
// the n-1 denominator, z = (x - mean) / sd, missing samples as 0 so that a product with
// a missing sample contributes nothing -- the reference's pairwise NaN skip,
// corHelper.cu:101) into the FP64 copy Z or, for the tensor-core Gram, into the
// split-BF16 operands (and z as an FP32 pair for the FP64 re-tests); the FP64
// correlation is the tiled Gram C = Z^T Z / (n - 1) over upper-triangle 8 x 8 tiles,
// mirrored on write.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "internal.cuh"

namespace cg = cooperative_groups;

namespace hpc {
namespace {

constexpr int kStdThreads = 256;

// Error-free FP32 sum (Knuth's TwoSum): a + b == s + e exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// x - mean as an unevaluated FP32 pair (dh + de), mean = mh + ml; the pair is exact up
// to the representation error of ml (2^-48 |mean|).
__device__ __forceinline__ void centre_f32(float xv, float mh, float ml, float &dh, float &de) {
  float h, e;
  two_sum(xv, -mh, h, e);
  two_sum(h, e - ml, dh, de);
}

// Warp sum of FP32 pairs (h + l), compensated: every lane ends with the total.
__device__ __forceinline__ void warp_sum_pair(float &h, float &l) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
    float s, e;
    two_sum(h, oh, s, e);
    h = s;
    l = l + ol + e;
  }
}

// The scalars of one variable that the sample loops use, formed once per block by thread
// 0 (an FP64 division or square root is a long instruction sequence on this GPU's
// 1/64-rate FP64 pipe: in every thread of every block they would cost more than the
// sample loops). mean and inv_sd = 1 / sd in FP64; scale = 1 / sqrt(n - 1); FP32 pairs
// (h + l) of mean, inv_sd * scale (i*) and inv_sd (j*).
struct ColScalars {
  double mean, inv_sd, scale;
  float mh, ml, ih, il, jh, jl;
};

// Block-wide total of the warps' FP32 pairs (lane 0 of warp w stored them in rh[w],
// rl[w]), compensated in FP32, converted to FP64 once: thread 0 only. (Every FP64 warp
// instruction occupies the SM's FP64 unit for 16 cycles, whether one lane or 32 use it.)
__device__ __forceinline__ double warp_totals(const float *rh, const float *rl) {
  float h = 0.f, l = 0.f;
#pragma unroll
  for (int w = 0; w < kStdThreads / 32; ++w) {
    float s, e;
    two_sum(h, rh[w], s, e);
    h = s;
    l += rl[w] + e;
  }
  return (double)h + (double)l;
}
__device__ __forceinline__ double warp_totals(const double *red) {
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kStdThreads / 32; ++w) t += red[w];
  return t;
}

__device__ __forceinline__ void finish_scalars(double ss, long long n, int ref_compat, ColScalars &S) {
  // z = (x - mean) * (1 / sd): one multiply per sample instead of a division; 1 / sd by
  // rsqrt of the variance (within an ulp of 1 / sqrt, fewer FP64 instructions than a
  // square root and a division)
  if (ref_compat)  // corHelper.cu:75: sqrtf of (sum / (dim - 1.f))
    S.inv_sd = 1.0 / (double)sqrtf((float)(ss / (double)((float)n - 1.f)));
  else
    S.inv_sd = rsqrt(ss / (double)(n - 1));
  const double denom = ref_compat ? (double)((float)n - 1.f) : (double)(n - 1);
  S.scale = rsqrt(denom);
  const double inv = S.inv_sd * S.scale;
  S.ih = (float)inv;
  S.il = (float)(inv - (double)S.ih);
  S.jh = (float)S.inv_sd;
  S.jl = (float)(S.inv_sd - (double)S.jh);
}

// Column moments of FP32 samples with FP64-grade accuracy but FP32 arithmetic per sample
// (these loops touch every sample): compensated FP32 sums per thread and warp (TwoSum),
// the warps' pairs added in FP64. NaN samples are skipped, as cpuMeans / the reference's
// SD loop skip them.
__device__ __forceinline__ void column_scalars(const float *__restrict__ x, long long n, int ref_compat,
                                               ColScalars &S) {
  __shared__ float rh[kStdThreads / 32], rl[kStdThreads / 32];
  __shared__ long long redc[kStdThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float sh = 0.f, sl = 0.f;
  int cnt = 0;
  for (long long k = threadIdx.x; k < n; k += kStdThreads) {
    const float xv = x[k];
    if (xv == xv) {
      float s, e;
      two_sum(sh, xv, s, e);
      sh = s;
      sl += e;
      ++cnt;
    }
  }
  warp_sum_pair(sh, sl);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) {
    rh[wid] = sh;
    rl[wid] = sl;
    redc[wid] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long c = 0;
    for (int w = 0; w < kStdThreads / 32; ++w) c += redc[w];
    S.mean = warp_totals(rh, rl) / (double)c;
    S.mh = (float)S.mean;
    S.ml = (float)(S.mean - (double)S.mh);
  }
  __syncthreads();
  const float mh = S.mh, ml = S.ml;
  float qh = 0.f, ql = 0.f;
  for (long long k = threadIdx.x; k < n; k += kStdThreads) {
    const float xv = x[k];
    if (xv == xv) {
      float dh, de;
      centre_f32(xv, mh, ml, dh, de);
      const float p = dh * dh;
      float pe = fmaf(dh, dh, -p);  // exact error of the square
      pe = fmaf(2.f * dh, de, pe);
      pe = fmaf(de, de, pe);
      float s, e;
      two_sum(qh, p, s, e);
      qh = s;
      ql += e + pe;
    }
  }
  warp_sum_pair(qh, ql);
  __syncthreads();  // rh, rl are reused
  if (lane == 0) {
    rh[wid] = qh;
    rl[wid] = ql;
  }
  __syncthreads();
  if (threadIdx.x == 0) finish_scalars(warp_totals(rh, rl), n, ref_compat, S);
  __syncthreads();
}

// FP64 samples: FP64 sums (two passes, as the reference's mean-then-SD loops)
__device__ __forceinline__ void column_scalars(const double *__restrict__ x, long long n, int ref_compat,
                                               ColScalars &S) {
  __shared__ double red[kStdThreads / 32];
  __shared__ long long redc[kStdThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double s = 0.0;
  int cnt = 0;
  for (long long k = threadIdx.x; k < n; k += kStdThreads) {
    const double xv = x[k];
    if (!isnan(xv)) {
      s += xv;
      ++cnt;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) {
    red[wid] = s;
    redc[wid] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long c = 0;
    for (int w = 0; w < kStdThreads / 32; ++w) c += redc[w];
    S.mean = warp_totals(red) / (double)c;
    S.mh = (float)S.mean;
    S.ml = (float)(S.mean - (double)S.mh);
  }
  __syncthreads();
  const double mean = S.mean;
  double q = 0.0;
  for (long long k = threadIdx.x; k < n; k += kStdThreads) {
    const double xv = x[k];
    if (!isnan(xv)) {
      const double d = xv - mean;
      q = fma(d, d, q);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  __syncthreads();
  if (lane == 0) red[wid] = q;
  __syncthreads();
  if (threadIdx.x == 0) finish_scalars(warp_totals(red), n, ref_compat, S);
  __syncthreads();
}

// Outputs of the standardisation (compile-time, so that no sample loop carries a
// branch or an idle computation for an absent output):
//   kStdZ        Z: FP64 standardised samples
//   kStdSplitZ   Z and the split-BF16 planes of the tensor-core Gram (FP64 samples)
//   kStdSplitPair the split-BF16 planes and z as an unevaluated FP32 pair (zh + zl,
//                FP64-grade), formed with no FP64 instruction per sample (FP32 samples)
constexpr int kStdZ = 0, kStdSplitZ = 1, kStdSplitPair = 2;

// z = (x - mean) * inv as an FP32 pair from the centred pair (dh + de) and inv = ih + il:
// the product's rounding error is recovered exactly (fmaf), the cross terms are 2^-24
// of the result
__device__ __forceinline__ void scale_pair(float dh, float de, float ih, float il, float &zh, float &zl) {
  const float p = dh * ih;
  float e = fmaf(dh, ih, -p);
  e = fmaf(dh, il, fmaf(de, ih, e));
  zh = p + e;
  zl = e - (zh - p);
}

// grid: one block per variable of every instance (flattened over row_prefix).
template <typename TIn, int OUT>
__global__ void __launch_bounds__(kStdThreads) standardise_kernel(const TIn *__restrict__ X, StdArgs a,
                                                                  double *__restrict__ Z, float *__restrict__ ZP,
                                                                  long long zp_plane, __nv_bfloat16 *__restrict__ P) {
  constexpr bool kF32 = std::is_same<TIn, float>::value;
  static_assert(OUT != kStdSplitPair || kF32, "the FP32 pair output is formed from FP32 samples");
  const long long t = blockIdx.x;
  const int b = find_inst(a.row_prefix, a.count, t);
  const long long v = t - a.row_prefix[b];
  const long long n = a.n[b];
  const TIn *x = X + a.x_off[b] + v * n;
  __shared__ ColScalars S;
  column_scalars(x, n, a.ref_compat, S);
  const double mean = S.mean, inv_sd = S.inv_sd;
  if constexpr (OUT == kStdZ) {
    double *z = Z + a.z_off[b] + v * n;
    for (long long k = threadIdx.x; k < n; k += kStdThreads) {
      const double xv = (double)x[k];
      z[k] = isnan(xv) ? 0.0 : (xv - mean) * inv_sd;
    }
    return;
  }
  // split-BF16 operand of the tensor-core Gram: two planes T = [hi | lo] of
  // zs = z / sqrt(n - 1) (the Gram's producer pairs the planes: hi.hi + hi.lo + lo.hi +
  // lo.lo is the correlation). hi = bf16(zs), lo = bf16(zs - hi), the subtraction exact in
  // FP32. FP32 samples form zs in FP32 pairs (x - mean as dh + de, times 1 / sqrt(n - 1)
  // / sd as ih + il): within an ulp of the FP64 value. Two consecutive samples per
  // thread, so that the planes are written as 4-byte pairs.
  const double scale = S.scale;
  const float mh = S.mh, ml = S.ml, ih = S.ih, il = S.il, jh = S.jh, jl = S.jl;
  const long long n_pad = a.n_pad[b], K = a.kdim[b];
  __nv_bfloat16 *pr = P + a.tc_off[b] + v * K;
  double *z = OUT == kStdSplitZ ? Z + a.z_off[b] + v * n : nullptr;
  float *zh = OUT == kStdSplitPair ? ZP + a.z_off[b] + v * n : nullptr;
  float *zl = OUT == kStdSplitPair ? zh + zp_plane : nullptr;
  for (long long k = 2 * (long long)threadIdx.x; k < n_pad; k += 2 * kStdThreads) {
    float s2[2] = {0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long kk = k + u;
      if (kk >= n) break;
      if constexpr (kF32) {
        const float xv = x[kk];
        float dh = 0.f, de = 0.f;
        if (xv == xv) centre_f32(xv, mh, ml, dh, de);
        s2[u] = fmaf(dh, ih, fmaf(dh, il, de * ih));
        if constexpr (OUT == kStdSplitPair) {
          float h, l;
          scale_pair(dh, de, jh, jl, h, l);
          zh[kk] = h;
          zl[kk] = l;
        } else {
          z[kk] = xv != xv ? 0.0 : ((double)xv - mean) * inv_sd;
        }
      } else {
        const double xv = x[kk];
        const double zv = isnan(xv) ? 0.0 : (xv - mean) * inv_sd;
        z[kk] = zv;
        s2[u] = (float)(zv * scale);
      }
    }
    const __nv_bfloat162 hi = __floats2bfloat162_rn(s2[0], s2[1]);
    const float2 hf = __bfloat1622float2(hi);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(s2[0] - hf.x, s2[1] - hf.y);
    *reinterpret_cast<__nv_bfloat162 *>(pr + k) = hi;
    *reinterpret_cast<__nv_bfloat162 *>(pr + n_pad + k) = lo;
  }
}

// FP64 standardised samples from the FP32 pairs (zh + zl, exact in FP64)
__global__ void pair_to_f64_kernel(const float *__restrict__ zh, const float *__restrict__ zl, long long count,
                                   double *__restrict__ Z) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
    Z[i] = (double)zh[i] + (double)zl[i];
}

// FP64 Gram of the standardised data over the upper triangle of 8 x 8 output tiles.
//
// Bound: the FP64 pipe, 2 FMA per clock per SM here -- so slow that a warp's FMA leaves
// room for 16 cycles of other work, and register tiling buys nothing. What counts is that
// every SM has its share: a tile is small (8 x 8: the triangle's waste is below 8 / p, a
// problem of 50 variables has 28 tiles), its samples are dealt to kGramSlices slices of a
// block and, where the tiles alone do not fill the GPU, to the blocks of a cluster, which
// add their partial sums through distributed shared memory in a fixed order (no
// workspace, no atomics, results do not depend on timing). With one 64 x 64 tile per block
// and no split a problem of 50 variables ran on one SM. Before and after, whole calls: the
// allocation-free correlation of p = 96, n = 1500 1586 -> 38 us (its floor is 12 us of FP64
// pipe), a skeleton of p = 50, n = 1000 from observations 1287 -> 241 us, the plain FP64 path
// at p = 300, n = 1500 1878 -> 391 us (floor of its Gram 117 us).
constexpr int BM = 8, BK = 64, GT = 256;
constexpr int kGramSlices = GT / (BM * BM);  // samples k % 4 of a stage go to slice k % 4
constexpr int kGramMaxSplit = 8;             // portable cluster size

__global__ void __launch_bounds__(GT) gram_f64_kernel(const double *__restrict__ Zall, double *__restrict__ Call,
                                                      GramArgs g, int split) {
  const long long tt = blockIdx.x / split;
  const int part = (int)(blockIdx.x - tt * split);  // = the block's rank in its cluster
  const int b = find_inst(g.tile_prefix, g.count, tt);
  const long long t = tt - g.tile_prefix[b];
  const long long p = g.p[b], n = g.n[b];
  const double *__restrict__ Z = Zall + g.z_off[b];
  double *__restrict__ C = Call + g.c_off[b];
  // (bi, bj), bi <= bj, column by column of the triangle of tiles: an FP32 estimate of the
  // triangular root, corrected in integers
  long long bj = (long long)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  if (bj < 0) bj = 0;
  while (bj > 0 && bj * (bj + 1) / 2 > t) --bj;
  while ((bj + 1) * (bj + 2) / 2 <= t) ++bj;
  const long long bi = t - bj * (bj + 1) / 2;
  const long long a0 = bi * BM, b0 = bj * BM;
  // two operands of BM columns, column c of a stage at [k][c]; the padded row of 9 doubles
  // keeps the stores (consecutive k) free of bank conflicts
  __shared__ double s_op[2][BK][BM + 1];
  __shared__ double s_sum[GT];
  const int tid = threadIdx.x;
  const int slice = tid / (BM * BM), out = tid % (BM * BM), r = out / BM, c = out % BM;
  // this block's samples: whole stages, so that the parts differ by one stage at most
  const long long stages = (n + BK - 1) / BK;
  const long long k_lo = (stages * part / split) * BK, k_hi = min(n, (stages * (part + 1) / split) * BK);
  constexpr int kLoads = 2 * BM * BK / GT;  // values per thread and stage
  double reg[kLoads];
  auto fetch = [&](long long k0) {
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = tid + q * GT, col = idx / BK, kk = idx % BK;  // col: 0..7 of A, 8..15 of B
      const long long v = col < BM ? a0 + col : b0 + (col - BM), k = k0 + kk;
      reg[q] = (v < p && k < k_hi) ? Z[v * n + k] : 0.0;
    }
  };
  double acc = 0.0;
  if (k_lo < k_hi) fetch(k_lo);
  for (long long k0 = k_lo; k0 < k_hi; k0 += BK) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = tid + q * GT, col = idx / BK, kk = idx % BK;
      s_op[col / BM][kk][col % BM] = reg[q];
    }
    __syncthreads();
    if (k0 + BK < k_hi) fetch(k0 + BK);  // the next stage's loads overlap this one's FMAs
#pragma unroll 4
    for (int kk = slice; kk < BK; kk += kGramSlices) acc = fma(s_op[0][kk][r], s_op[1][kk][c], acc);
  }
  s_sum[tid] = acc;
  __syncthreads();
  if (tid < BM * BM) {
    double v = s_sum[tid];
#pragma unroll
    for (int q = 1; q < kGramSlices; ++q) v += s_sum[tid + q * BM * BM];
    s_sum[tid] = v;
  }
  if (split > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (part == 0 && tid < BM * BM) {
      double v = s_sum[tid];
      for (int q = 1; q < split; ++q) v += cluster.map_shared_rank(s_sum, q)[tid];
      acc = v;
    }
    cluster.sync();  // no block leaves while its sums are read
    if (part != 0) return;
  } else {
    acc = s_sum[tid];
  }
  if (tid < BM * BM) {
    const long long ra = a0 + r, cb = b0 + c;
    if (ra < p && cb < p && ra <= cb) {
      const double v = acc / g.denom[b];
      C[ra * p + cb] = v;
      C[cb * p + ra] = v;
    }
  }
}

// Blocks a tile's samples are split over: the smallest power of two that gives every SM
// four blocks (the FP64 pipe is shared by the SM's blocks, so the last wave is at most a
// quarter of a block's work long), up to a portable cluster.
int gram_split(long long total_tiles) {
  int split = 1;
  while (split < kGramMaxSplit && total_tiles * split < 152LL * 4) split *= 2;
  return split;
}

__global__ void to_f32_kernel(const double *__restrict__ C, int64_t count, float *__restrict__ C32) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    C32[i] = (float)C[i];
}

}  // namespace

long long gram_f64_tiles(int64_t p) {
  const long long nb = (p + BM - 1) / BM;
  return nb * (nb + 1) / 2;
}

hpc_status launch_standardise(const void *X, bool f32, const StdArgs &a, long long total_rows, double *Z,
                              float *ZP, long long zp_plane, __nv_bfloat16 *P, cudaStream_t s) {
  const unsigned grid = (unsigned)total_rows;
  if (!P) {
    if (!Z) return HPC_ERR_INVALID_ARG;
    if (f32)
      standardise_kernel<float, kStdZ><<<grid, kStdThreads, 0, s>>>((const float *)X, a, Z, nullptr, 0, nullptr);
    else
      standardise_kernel<double, kStdZ><<<grid, kStdThreads, 0, s>>>((const double *)X, a, Z, nullptr, 0, nullptr);
  } else if (ZP) {
    if (!f32) return HPC_ERR_INVALID_ARG;
    standardise_kernel<float, kStdSplitPair><<<grid, kStdThreads, 0, s>>>((const float *)X, a, nullptr, ZP, zp_plane, P);
  } else {
    if (!Z) return HPC_ERR_INVALID_ARG;
    if (f32)
      standardise_kernel<float, kStdSplitZ><<<grid, kStdThreads, 0, s>>>((const float *)X, a, Z, nullptr, 0, P);
    else
      standardise_kernel<double, kStdSplitZ><<<grid, kStdThreads, 0, s>>>((const double *)X, a, Z, nullptr, 0, P);
  }
  HPC_LAUNCH_CHECK("standardise_kernel");
  return HPC_OK;
}

hpc_status launch_pair_to_f64(const float *zh, const float *zl, long long count, double *Z, cudaStream_t s) {
  pair_to_f64_kernel<<<1024, 256, 0, s>>>(zh, zl, count, Z);
  HPC_LAUNCH_CHECK("pair_to_f64_kernel");
  return HPC_OK;
}

hpc_status launch_gram_f64(const double *Z, double *C, const GramArgs &a, long long total_tiles, cudaStream_t s) {
  const int split = gram_split(total_tiles);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(total_tiles * split));
  cfg.blockDim = dim3(GT);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HPC_CUDA(cudaLaunchKernelEx(&cfg, gram_f64_kernel, Z, C, a, split));
  return HPC_OK;
}

hpc_status launch_to_f32(const double *C, int64_t count, float *C32, cudaStream_t s) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 152 * 16));
  to_f32_kernel<<<blocks, 256, 0, s>>>(C, count, C32);
  HPC_LAUNCH_CHECK("to_f32_kernel");
  return HPC_OK;
}

}  // namespace hpc
