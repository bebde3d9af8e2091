// Level-l CI tests (l >= 1): the re-test and record kernels, the level-kernel
// instantiations of levels 1-8 and the launchers (the level kernels' device code is in
// citest.cuh, wide.cuh and level_kernel.cuh).
#include <algorithm>
#include <atomic>

#include "level_kernel.cuh"

namespace hpc {
namespace {

// p-values of the removals decided in FP32 (negative pmax), for every instance's
// records: FP64 re-evaluation where the instance has an FP64 matrix -- a result below
// alpha flags kErrBandViolation (the FP32 error bound did not hold) -- else the formula
// in FP32 on the stored FP32 |r|. Run at the end of every skeleton run. The instances
// run side by side, a group of gridDim / count blocks (at least one) each: taking them
// one after another over the whole grid cost a chain of dependent loads per instance
// (0.8 ms for a batch of 512 instances of p 20-800).
__global__ void finalize_records_kernel(const Inst *__restrict__ inst, int count) {
  if (count <= 0) return;
  const unsigned per = max(1u, gridDim.x / (unsigned)count);  // blocks per instance
  const unsigned groups = gridDim.x / per;
  const unsigned long long tid = (blockIdx.x % per) * (unsigned long long)blockDim.x + threadIdx.x;
  const unsigned long long nthreads = (unsigned long long)per * blockDim.x;
  for (int b = (int)(blockIdx.x / per); b < count; b += (int)groups) {
    const Inst &I = inst[b];
    unsigned long long end = I.g->rec_count;
    if (end > (unsigned long long)I.rec_cap) end = (unsigned long long)I.rec_cap;
    for (unsigned long long r = tid; r < end; r += nthreads) {
      int32_t *rec = I.recs + r * (unsigned long long)I.rec_stride;
      RecHead *h = reinterpret_cast<RecHead *>(rec);
      if (!(h->pmax < 0.0)) continue;
      if (!I.cor64) {
        h->pmax = (double)calc_pvalue32((float)(-1.0 - h->pmax), I.n_obs);
        continue;
      }
      // level 1: the closed form from the three entries (what exact_pvalue evaluates
      // there, without its matrix in local memory); else the general path, its arrays
      // sized by the level
      double pv;
      const int l = h->level;
      if (l == 1) {
        const int64_t k = rec[kRecHeadWords];
        pv = pval_l1_64(I.cor64[h->i * I.p + h->j], I.cor64[h->i * I.p + k], I.cor64[h->j * I.p + k], I.n_obs);
      } else {
        // most records above level 1 are of levels 2-4: in registers, since the general path
        // keeps its matrices in local memory and a thread steps through them alone (skeletons of
        // p = 50 and of p = 300 in FP64, whole calls: 241 -> 236 and 391 -> 378 us; with tens of
        // thousands of level-1 records the FP64 pipe bounds the kernel, not this)
        bool nan_p = false, ok = false;
        double r = 0.0;
        if (l <= 4) r = partial_r_registers<4>(I, h->i, h->j, rec + kRecHeadWords, l, &nan_p, &ok);
        if (ok)
          pv = nan_p ? nan("") : calc_pvalue64(r, I.n_obs);
        else
          pv = l <= 16 ? exact_pvalue<16>(I, h->i, h->j, rec + kRecHeadWords, l)
                       : exact_pvalue<HPC_MAX_LEVEL>(I, h->i, h->j, rec + kRecHeadWords, l);
      }
      h->pmax = pv;
      if (!(pv >= I.alpha)) atomicOr(&I.g->err, kErrBandViolation);
    }
  }
}

// Records of all instances compacted into one buffer: one warp per record, its
// words copied by the lanes (record r of the output belongs to the instance b with
// prefix[b] <= r < prefix[b + 1]).
__global__ void gather_records_kernel(const Inst *__restrict__ inst, int count, const long long *__restrict__ prefix,
                                      long long total, int stride, int32_t *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < total; r += nw) {
    const int b = find_inst(prefix, count, r);
    const int32_t *src = inst[b].recs + (r - prefix[b]) * (long long)stride;
    for (int w = lane; w < stride; w += 32) out[r * (long long)stride + w] = src[w];
  }
}

// Records of all instances in the packed form of hpc_batch_get_records_packed. The host
// cuts them into segments, one per (instance, level) with removals: an instance's
// records are appended level by level, so a segment is a contiguous run of `count`
// records from record `src` of instance `inst` (rec_stride words each), and it goes to
// the contiguous words from `dst`, w = 6 + 2 ceil(l / 2) words per record (head, l ids,
// -1 padding). One block per segment, its threads over the segment's output words
// (coalesced writes, no per-record search).
__global__ void pack_records_kernel(const Inst *__restrict__ inst, const RecSegment *__restrict__ seg, int nseg,
                                    int32_t *__restrict__ out) {
  for (int g = blockIdx.x; g < nseg; g += gridDim.x) {
    const RecSegment S = seg[g];
    const Inst &I = inst[S.inst];
    const int l = S.level;
    const int w = 6 + ((l + 1) & ~1);
    const long long words = S.count * (long long)w;
    const int32_t *src = I.recs + S.src * (long long)I.rec_stride;
    int32_t *dst = out + S.dst;
    for (long long t = threadIdx.x; t < words; t += blockDim.x) {
      const long long r = t / w;
      const int q = (int)(t - r * w);
      dst[t] = q < 6 + l ? src[r * I.rec_stride + q] : -1;
    }
  }
}

// samples [k0, end) of the product of two standardised columns
__device__ __forceinline__ double warp_dot(const Inst &I, int64_t a, int64_t b, int64_t k0, int64_t end) {
  const int lane = threadIdx.x & 31;
  double s = zdot(I, a, b, k0 + lane, 32, end);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__device__ __forceinline__ double warp_dot(const Inst &I, int64_t a, int64_t b) { return warp_dot(I, a, b, 0, I.n_z); }

// FP64 re-tests deferred by the level kernels (instances without an FP64 matrix). A
// re-test of level l needs the E = (l + 2)(l + 1) / 2 FP64 correlation entries among
// i, j and S, each a dot product of two FP64-standardised columns (n samples). One warp
// per dot product: the launch's first W items (W = min(queued, rq_vcap / E)) are cut
// into W * E (item, entry) units over the grid, each warp writes its entry to the item's
// scratch row and counts it done; the warp completing an item's last entry gathers the
// row into its (l + 2)^2 matrix in shared memory and lane 0 evaluates the reference
// formula. So a level with a few re-tests of many entries (the high levels) runs them
// side by side instead of one warp stepping through 100+ dot products; items beyond the
// scratch take a warp each. Level-0 items (one entry) set the kept bits of both
// triangles; level >= 1 items remove the edge. The done counters return to zero when
// their item is evaluated, ready for the next launch.
// With few items the samples of a dot product are cut into up to kRetestParts parts of a warp each
// (a warp alone goes over 8000 samples in about 20 us, and most levels of a deep skeleton have a
// handful of re-tests): the warp completing the item adds up the parts, in their order.
// KM: the highest level of the launch's items (16 for levels up to 16, HPC_MAX_LEVEL
// above), which sizes the FP64 fallback's local arrays.
constexpr int kRetestWarps = 8;
constexpr int kRetestParts = 8;

// the variable at position r of a re-test's matrix order (i, j, S)
__device__ __forceinline__ int64_t retest_var(const RetestItem *it, int r) {
  return r == 0 ? (int64_t)it->i : r == 1 ? (int64_t)it->j : (int64_t)it->ids[r - 2];
}

// entry e of the upper triangle of a k x k matrix, row by row: (r, c), r < c
__device__ __forceinline__ void entry_rc(int e, int k, int &r, int &c) {
  r = 0;
  while (e >= k - 1 - r) {
    e -= k - 1 - r;
    ++r;
  }
  c = r + 1 + e;
}

// partial_r_of_matrix by the whole warp, M in shared memory (left as it was where *ok is false, which
// is where it takes the pseudoinverse): a lane per member, column by column of the factor, every
// entry in the same operations and order -- so the same value. One lane alone steps through
// l^3 / 6 dependent FP64 operations, about 80 us at level 12, longer than all the dot products
// of a level with a few re-tests. The factor goes to the lower triangle of the S block, w_i and
// w_j to the first two columns; the upper triangle keeps the entries.
__device__ __forceinline__ double warp_partial_r(double *M, int l, bool *nan_p, bool *ok) {
  const int lane = threadIdx.x & 31, k = l + 2;
  bool bad = false;
  for (int q = lane; q < k * k; q += 32) bad |= isnan(M[q]);
  *nan_p = __any_sync(0xffffffffu, bad);
  *ok = true;
  if (*nan_p) return 0.0;
  double *row = M + (lane + 2) * k;  // lane < l: its member's row
  double d = 1.0, vx = lane < l ? M[lane + 2] : 0.0, vy = lane < l ? M[k + lane + 2] : 0.0;
  for (int c = 0; c < l; ++c) {
    if (!__shfl_sync(0xffffffffu, d > 1e-10, c)) {
      *ok = false;
      break;
    }
    if (lane == c) {
      const double lcc = sqrt(d);
      row[c + 2] = lcc;
      row[0] = vx / lcc;
      row[1] = vy / lcc;
    }
    __syncwarp();
    if (lane > c && lane < l) {
      const double *rc = M + (c + 2) * k;
      double v = rc[lane + 2];
      for (int q = 0; q < c; ++q) v -= row[q + 2] * rc[q + 2];
      v /= rc[c + 2];
      row[c + 2] = v;
      d -= v * v;
      vx -= v * rc[0];
      vy -= v * rc[1];
    }
    __syncwarp();
  }
  double r = 0.0;
  if (*ok) {
    double ax = 1.0, ay = 1.0, b = M[1];
    for (int q = 0; q < l; ++q) {
      const double wx = M[(q + 2) * k], wy = M[(q + 2) * k + 1];
      ax -= wx * wx;
      ay -= wy * wy;
      b -= wx * wy;
    }
    *ok = ax > 1e-10 && ay > 1e-10;
    r = b / sqrt(ax * ay);
  }
  if (!*ok) {  // the matrix as it was
    __syncwarp();
    for (int q = lane; q < k * k; q += 32) {
      const int a = q / k, c = q - a * k;
      if (a > c) M[q] = M[c * k + a];
      if (a == c) M[q] = 1.0;
    }
    __syncwarp();
  }
  return r;
}

// The FP64 decision of item it from its matrix M (k x k, warp-filled); whole warp.
template <int KM>
__device__ __forceinline__ void retest_decide(const Launch &L, const Inst &I, const RetestItem *it, int l, double *M) {
  const int lane = threadIdx.x & 31;
  bool nan_p = false, ok = false;
  double r = 0.0;
  if (l > 1) r = warp_partial_r(M, l, &nan_p, &ok);
  if (lane == 0) {
    if (!ok) r = partial_r_of_matrix<KM>(M, l, &nan_p);
    double pv;
    const int64_t i = it->i, j = it->j;
    if (decide_of_r(I, r, nan_p, &pv) && claim_edge(I, i, j)) write_record(I, L.level, i, j, it->ids, l, pv);
  }
}

// Levels 1-4 (K = l + 2 <= 6 variables): one warp per item, every lane accumulating the
// E = K(K - 1) / 2 products over its samples (k = lane, lane + 32, ...) in passes of
// kRetestPass entries (the accumulators of a pass stay in registers), so that each of
// the K columns is read once per item instead of once per entry it takes part in (2E
// column reads in the entry-parallel form). Above level 4 the entry-parallel form is
// faster (measured on a batch of 512 instances of p 20-800: a re-test's 28-45 entries
// spread over as many warps beat one warp stepping through the columns, and the column
// form's registers halve occupancy). The products are
// summed as in zdot: the FP32 pairs' products with their exact rounding errors and cross
// terms, compensated in FP32 and carried into FP64 every 16 samples of a lane.
constexpr int kRetestPass = 16;
constexpr int kColumnTop = 4;  // the highest level re-tested by columns

// (r, c) of entry e of the upper triangle of a K x K matrix, row by row
__host__ __device__ constexpr int entry_row(int e, int K) {
  int r = 0;
  while (e >= K - 1 - r) {
    e -= K - 1 - r;
    ++r;
  }
  return r;
}
__host__ __device__ constexpr int entry_col(int e, int K) {
  int r = 0;
  while (e >= K - 1 - r) {
    e -= K - 1 - r;
    ++r;
  }
  return r + 1 + e;
}

// one pass: entries E0 .. E0 + EN - 1, written to the warp's matrix M (K x K) by lane 0
template <int K, int E0, int EN>
__device__ __forceinline__ void retest_columns_pass(const Inst &I, const float *const *ch, int64_t lo_off,
                                                    double *M) {
  const int lane = threadIdx.x & 31;
  const int64_t n = I.n_z;
  double acc[EN];
#pragma unroll
  for (int e = 0; e < EN; ++e) acc[e] = 0.0;
  for (int64_t k0 = lane; k0 < n; k0 += 32 * 16) {
    float sh[EN], sl[EN];
#pragma unroll
    for (int e = 0; e < EN; ++e) sh[e] = sl[e] = 0.f;
    // the products of one sample's loaded values
    auto add = [&](const float *ah, const float *al) {
      int e = 0;
#pragma unroll
      for (int r = 0; r < K; ++r)
#pragma unroll
        for (int c = r + 1; c < K; ++c, ++e) {
          if (e < E0 || e >= E0 + EN) continue;
          const int x = e - E0;
          const float p = ah[r] * ah[c];
          float er = fmaf(ah[r], ah[c], -p);
          er = fmaf(ah[r], al[c], fmaf(al[r], ah[c], er));
          const float t = sh[x] + p;
          const float bb = t - sh[x];
          sl[x] += ((sh[x] - (t - bb)) + (p - bb)) + er;
          sh[x] = t;
        }
    };
    // S samples at a time, all loaded before the arithmetic (no bounds test between):
    // the loop is bound by its round trips to memory, so a round trip carries as many
    // samples as the registers allow
    constexpr int S = K <= 4 ? 8 : K == 5 ? 4 : 2;
#pragma unroll 1
    for (int u = 0; u < 16; u += S) {
      const int64_t k = k0 + 32 * u;
      if (k + 32 * (S - 1) < n) {
        float ah[S][K], al[S][K];
#pragma unroll
        for (int v = 0; v < S; ++v)
#pragma unroll
          for (int r = 0; r < K; ++r) {
            ah[v][r] = ch[r][k + 32 * v];
            al[v][r] = ch[r][k + 32 * v + lo_off];
          }
#pragma unroll
        for (int v = 0; v < S; ++v) add(ah[v], al[v]);
      } else {
#pragma unroll 1
        for (int v = 0; v < S && k + 32 * v < n; ++v) {  // the ragged end, a sample at a time
          float ah[K], al[K];
#pragma unroll
          for (int r = 0; r < K; ++r) {
            ah[r] = ch[r][k + 32 * v];
            al[r] = ch[r][k + 32 * v + lo_off];
          }
          add(ah, al);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < EN; ++e) acc[e] += (double)sh[e] + (double)sl[e];
  }
#pragma unroll
  for (int e = 0; e < EN; ++e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if (lane == 0) {
      const int r = entry_row(E0 + e, K), c = entry_col(E0 + e, K);
      M[r * K + c] = M[c * K + r] = acc[e] / I.denom;
    }
  }
}

template <int K, int E0>
__device__ __forceinline__ void retest_columns_passes(const Inst &I, const float *const *ch, int64_t lo_off,
                                                      double *M) {
  constexpr int E = K * (K - 1) / 2;
  if constexpr (E0 < E) {
    constexpr int EN = E - E0 < kRetestPass ? E - E0 : kRetestPass;
    retest_columns_pass<K, E0, EN>(I, ch, lo_off, M);
    retest_columns_passes<K, E0 + kRetestPass>(I, ch, lo_off, M);
  }
}

// the item's matrix M (K x K, the warp's shared memory) from its columns
template <int K>
__device__ __forceinline__ void retest_item_columns(const Inst &I, const RetestItem *it, double *M) {
  constexpr int E = K * (K - 1) / 2;
  static_assert(E <= 32, "one lane per entry");
  const int lane = threadIdx.x & 31;
  const int64_t n = I.n_z;
  if (lane < K) M[lane * K + lane] = 1.0;
  // lane e: entry e -- formed by an earlier re-test? then no column is read
  int er = 0, ec = 0;
  int64_t va = 0, vb = 0;
  double v = 0.0;
  bool have = true;
  if (lane < E) {
    entry_rc(lane, K, er, ec);
    va = retest_var(it, er);
    vb = retest_var(it, ec);
    have = ecache_get(I, va, vb, &v);
  }
  if (__all_sync(0xffffffffu, have)) {
    if (lane < E) M[er * K + ec] = M[ec * K + er] = v;
    return;
  }
  const float *ch[K];
  const int64_t lo_off = I.zl - I.zh;  // the zl plane, at a fixed distance from zh
#pragma unroll
  for (int r = 0; r < K; ++r) ch[r] = I.zh + retest_var(it, r) * n;
  retest_columns_passes<K, 0>(I, ch, lo_off, M);
  __syncwarp();
  if (lane < E && !have) ecache_put(I, va, vb, M[er * K + ec]);
}

template <int KM>
__global__ void __launch_bounds__(kRetestWarps * 32, 2) retest_kernel(const __grid_constant__ Launch L) {
  extern __shared__ double retest_smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int l = L.level;
  const int k = l + 2;
  double *M = retest_smem + (size_t)wib * k * k;
  unsigned long long count = L.lc->rq_count;
  if (count > (unsigned long long)L.rq_cap) count = (unsigned long long)L.rq_cap;
  const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
  const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  if (l == 0) {
    for (unsigned long long q = warp; q < count; q += nwarps) {
      const RetestItem *it = L.rq + q;
      const Inst &I = *inst_of(L, it->inst);
      const int64_t i = it->i, j = it->j;
      double r;
      if (!ecache_get(I, i, j, &r)) {
        r = warp_dot(I, i, j) / I.denom;
        if (lane == 0) ecache_put(I, i, j, r);
      }
      double pv;
      if (lane == 0 && !decide_of_r(I, r, false, &pv)) {  // kept: both triangles' bits
        atomicOr(I.adj + i * I.W + (j >> 5), 1u << (j & 31));
        atomicOr(I.adj + j * I.W + (i >> 5), 1u << (i & 31));
      }
    }
    return;
  }
  const unsigned long long E = (unsigned long long)(k * (k - 1) / 2);
  // by columns once the items' entries would keep every warp busy: an item's columns take a warp
  // three (level 1) to eight (level 4) times as long as one entry does (30 items of level 4 in a batch
  // of 24: 134 us by columns, 34 us by entries in parts)
  const bool by_columns = l <= kColumnTop && count * E > nwarps;
  if (by_columns) {
    // an item per warp from its columns (instances with FP32-pair data; FP64 Z takes
    // the general path below)
    for (unsigned long long q = warp; q < count; q += nwarps) {
      const RetestItem *it = L.rq + q;
      const Inst &I = *inst_of(L, it->inst);
      if (!I.zh || !live_bit(I.adj, I.W, it->i, it->j)) continue;
      switch (l) {
        case 1: retest_item_columns<3>(I, it, M); break;
        case 2: retest_item_columns<4>(I, it, M); break;
        case 3: retest_item_columns<5>(I, it, M); break;
        default: retest_item_columns<6>(I, it, M); break;
      }
      __syncwarp();
      retest_decide<KM>(L, I, it, l, M);
      __syncwarp();
    }
  }
  // the items not taken above run entry by entry (the first W of them) or a warp each
  int parts = 1;
  while (L.rq_val && parts < kRetestParts && count * E * (unsigned)parts * 2 <= nwarps &&
         count * E * (unsigned)parts * 2 <= (unsigned long long)L.rq_vcap)
    parts *= 2;
  const unsigned long long EP = E * (unsigned)parts;  // scratch entries of an item
  const unsigned long long W = L.rq_val ? min(count, (unsigned long long)L.rq_vcap / EP) : 0ull;
  const unsigned long long units = W * EP;
  for (unsigned long long u = warp; u < units; u += nwarps) {
    const unsigned long long q = u / EP;
    const int x = (int)(u - q * EP), e = x / parts, part = x - e * parts;
    const RetestItem *it = L.rq + q;
    const Inst &I = *inst_of(L, it->inst);
    if (by_columns && I.zh) continue;  // decided above
    const int64_t i = it->i, j = it->j;
    if (live_bit(I.adj, I.W, i, j)) {  // else removed meanwhile: nothing to compute
      int r, c;
      entry_rc(e, k, r, c);
      const int64_t va = retest_var(it, r), vb = retest_var(it, c);
      double v;
      if (parts > 1) {  // (the parts of an entry do not look at the store: it may change between them)
        v = warp_dot(I, va, vb, I.n_z * part / parts, I.n_z * (part + 1) / parts);
      } else if (!ecache_get(I, va, vb, &v)) {
        v = warp_dot(I, va, vb) / I.denom;
        if (lane == 0) ecache_put(I, va, vb, v);
      }
      if (lane == 0) L.rq_val[u] = v;
    }
    unsigned last = 0;
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(L.rq_done + q, 1u) == (unsigned)(EP - 1);
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) continue;
    // the item's last entry: gather its matrix and decide
    __threadfence();
    if (lane == 0) L.rq_done[q] = 0u;
    if (!live_bit(I.adj, I.W, i, j)) continue;
    for (int t = lane; t < k * k; t += 32) {
      const int r = t / k, c = t - r * k;
      double v = 1.0;
      if (r != c) {
        const int a = r < c ? r : c, b2 = r < c ? c : r;
        const int eidx = a * k - a * (a + 1) / 2 + (b2 - a - 1);  // entry_rc's numbering
        const double *at = L.rq_val + q * EP + (unsigned)(eidx * parts);
        v = __ldcg(at);
        if (parts > 1) {
          for (int s = 1; s < parts; ++s) v += __ldcg(at + s);
          v /= I.denom;
          if (r < c) ecache_put(I, retest_var(it, r), retest_var(it, c), v);
        }
      }
      M[t] = v;
    }
    __syncwarp();
    retest_decide<KM>(L, I, it, l, M);
    __syncwarp();
  }
  // items beyond the scratch: a warp each
  for (unsigned long long q = W + warp; q < count; q += nwarps) {
    const RetestItem *it = L.rq + q;
    const Inst &I = *inst_of(L, it->inst);
    if (by_columns && I.zh) continue;                    // decided above
    if (!live_bit(I.adj, I.W, it->i, it->j)) continue;  // removed by another test meanwhile
    for (int r = 0; r < k; ++r) {
      if (lane == 0) M[r * k + r] = 1.0;
      for (int c2 = r + 1; c2 < k; ++c2) {
        const int64_t va = retest_var(it, r), vb = retest_var(it, c2);
        double v;
        if (!ecache_get(I, va, vb, &v)) {
          v = warp_dot(I, va, vb) / I.denom;
          if (lane == 0) ecache_put(I, va, vb, v);
        }
        if (lane == 0) M[r * k + c2] = M[c2 * k + r] = v;
      }
    }
    __syncwarp();
    retest_decide<KM>(L, I, it, l, M);
    __syncwarp();
  }
}

// Level-1 re-tests of instances with an FP64 matrix (mixed precision from a matrix or with the
// FP64-accurate Gram): a thread an item, the three entries read from the matrix, decided as
// tests_l1 decides them inline.
__global__ void __launch_bounds__(128) retest_matrix_kernel(const __grid_constant__ Launch L) {
  unsigned long long count = L.lc->rq_count;
  if (count > (unsigned long long)L.rq_cap) count = (unsigned long long)L.rq_cap;
  for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < count;
       q += (unsigned long long)gridDim.x * blockDim.x) {
    const RetestItem *it = L.rq + q;
    const Inst &I = *inst_of(L, it->inst);
    double pv;
    if (live_bit(I.adj, I.W, it->i, it->j) && exact_remove_fast<1>(I, it->i, it->j, it->ids, 1, &pv) &&
        claim_edge<false>(I, it->i, it->j))
      write_record(I, 1, it->i, it->j, it->ids, 1, pv);
  }
}

template <bool MIXED>
void *kernel_for(int level, int l1_variant) {
  if (MIXED && l1_variant == kSetOrder && level >= 2 && level <= kSetTop) {
    switch (level) {
      case 2: return (void *)level_kernel<2, true, kSetOrder>;
      case 3: return (void *)level_kernel<3, true, kSetOrder>;
      case 4: return (void *)level_kernel<4, true, kSetOrder>;
      case 5: return (void *)level_kernel<5, true, kSetOrder>;
      case 6: return (void *)level_kernel<6, true, kSetOrder>;
      case 7: return (void *)level_kernel<7, true, kSetOrder>;
      case 8: return (void *)level_kernel<8, true, kSetOrder>;
      default:
        return level <= 12 ? level_kernel_9_12(level, true, true)
               : level <= 16 ? level_kernel_13_16(level, true, true)
                             : level_kernel_17_24_set(level);
    }
  }
  switch (level) {
    case 1:
      if constexpr (MIXED) {
        if (l1_variant == kWide) return (void *)level_kernel<1, true, kWide>;
        if (l1_variant == (kWide | kQueueOnly)) return (void *)level_kernel<1, true, kWide | kQueueOnly>;
      }
      if (MIXED && l1_variant == (kL1Interleaved | kQueueOnly)) return (void *)level_kernel<1, true, kL1Interleaved | kQueueOnly>;
      if (MIXED && l1_variant == (kL1Prefetch | kQueueOnly)) return (void *)level_kernel<1, true, kL1Prefetch | kQueueOnly>;
      return l1_variant == kL1Chunked    ? (void *)level_kernel<1, MIXED, kL1Chunked>
             : l1_variant == kL1Prefetch ? (void *)level_kernel<1, MIXED, kL1Prefetch>
                                         : (void *)level_kernel<1, MIXED>;
    case 2:
      if constexpr (MIXED)
        if (l1_variant == kWide) return (void *)level_kernel<2, true, kWide>;
      return (void *)level_kernel<2, MIXED>;
    case 3: return (void *)level_kernel<3, MIXED>;
    case 4: return (void *)level_kernel<4, MIXED>;
    case 5: return (void *)level_kernel<5, MIXED>;
    case 6: return (void *)level_kernel<6, MIXED>;
    case 7: return (void *)level_kernel<7, MIXED>;
    case 8: return (void *)level_kernel<8, MIXED>;
    default:
      return level <= 12 ? level_kernel_9_12(level, MIXED, false)
                         : level <= 16 ? level_kernel_13_16(level, MIXED, false) : level_kernel_17_up(level, MIXED);
  }
}

// dynamic shared memory of a level kernel: the row offsets of own_scan (`rows` of them; none at
// level 1), the chunk of the wide level-1 body
int level_smem(int level, int variant, int rows) {
  if (level == 1) return (variant & kWide) ? (int)sizeof(Wide1Smem) : 0;
  return rows * (int)sizeof(unsigned long long);
}

}  // namespace

// Blocks of a level kernel that are resident at once. Asked of the driver once per device and
// kernel (a context asks for up to 60, which took a third of its creation).
int citest_grid(int precision, int level, int device, int l1_variant) {
  constexpr int kDevices = 64, kVariants = 16;
  static std::atomic<int> known[kDevices][2][HPC_MAX_LEVEL + 1][kVariants];
  const bool mixed = precision != HPC_PREC_FP64;
  std::atomic<int> *slot = device >= 0 && device < kDevices && l1_variant >= 0 && l1_variant < kVariants
                               ? &known[device][mixed ? 1 : 0][level][l1_variant] : nullptr;
  if (slot)
    if (const int g = slot->load(std::memory_order_acquire)) return g;
  void *k = mixed ? kernel_for<true>(level, l1_variant) : kernel_for<false>(level, l1_variant);
  const int smem = level_smem(level, l1_variant, kRowCache);  // the most it may have
  // beyond the default 48 KB of shared memory
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) cudaGetLastError();
  int per_sm = 0, sms = 0;
  bool ok = true;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem) != cudaSuccess || per_sm < 1) {
    per_sm = 1;
    ok = false;
  }
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 1) {
    sms = 1;
    ok = false;
  }
  if (slot && ok) slot->store(per_sm * sms, std::memory_order_release);
  return per_sm * sms;
}

// The re-test kernel of levels 17-32 needs up to 74 KB of dynamic shared memory, above
// the default 48 KB: allowed once per creation of a context that can reach those levels
// (not at launch, which may be under capture; levels up to 16 stay below 48 KB).
void retest_setup() {
  const int most = (int)(sizeof(double) * kRetestWarps * (HPC_MAX_LEVEL + 2) * (HPC_MAX_LEVEL + 2));
  if (cudaFuncSetAttribute((const void *)retest_kernel<HPC_MAX_LEVEL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           most) != cudaSuccess)
    cudaGetLastError();
}

hpc_status launch_retest(const Launch &L, int sms, cudaStream_t s) {
  const int kmax = L.level + 2;
  const size_t smem = sizeof(double) * (size_t)kRetestWarps * kmax * kmax;  // 20.7 KB at level 16
  if (L.level <= 16)
    retest_kernel<16><<<sms * 4, kRetestWarps * 32, smem, s>>>(L);
  else
    retest_kernel<HPC_MAX_LEVEL><<<sms * 4, kRetestWarps * 32, smem, s>>>(L);
  HPC_LAUNCH_CHECK("retest_kernel");
  return HPC_OK;
}

hpc_status launch_retest_matrix(const Launch &L, int sms, cudaStream_t s) {
  retest_matrix_kernel<<<sms * 2, 128, 0, s>>>(L);
  HPC_LAUNCH_CHECK("retest_matrix_kernel");
  return HPC_OK;
}

hpc_status launch_finalize_records(const Inst *inst, int count, cudaStream_t s) {
  finalize_records_kernel<<<152 * 4, 128, 0, s>>>(inst, count);
  HPC_LAUNCH_CHECK("finalize_records_kernel");
  return HPC_OK;
}

hpc_status launch_gather_records(const Inst *inst, int count, const long long *prefix, long long total, int stride,
                                 int32_t *out, cudaStream_t s) {
  if (total <= 0) return HPC_OK;
  const long long blocks = std::min<long long>((total + 7) / 8, 152 * 8);
  gather_records_kernel<<<(unsigned)blocks, 256, 0, s>>>(inst, count, prefix, total, stride, out);
  HPC_LAUNCH_CHECK("gather_records_kernel");
  return HPC_OK;
}

hpc_status launch_pack_records(const Inst *inst, const RecSegment *seg, int nseg, int32_t *out, cudaStream_t s) {
  if (nseg <= 0) return HPC_OK;
  pack_records_kernel<<<(unsigned)std::min(nseg, 152 * 16), 256, 0, s>>>(inst, seg, nseg, out);
  HPC_LAUNCH_CHECK("pack_records_kernel");
  return HPC_OK;
}

hpc_status launch_level(const Launch &L, int precision, int grid, int l1_variant, cudaStream_t s) {
  void *k = precision == HPC_PREC_FP64 ? kernel_for<false>(L.level, l1_variant)
                                       : kernel_for<true>(L.level, l1_variant);
  Launch args = L;
  if (l1_variant != kSetOrder && (l1_variant & kWide)) args.row_cache = 0;  // the wide-row kernels scan together
  void *params[] = {&args};
  // cooperative: every block co-resident, as the grid barriers require
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)level_smem(L.level, l1_variant, args.row_cache ? (int)L.inst0.p + 1 : 0);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HPC_CUDA(cudaLaunchKernelExC(&cfg, k, params));
  return HPC_OK;
}

}  // namespace hpc
