// CI tests of levels 1 and 2 on wide rows: rows whose neighbour lists hold hundreds to
// thousands of variables, as hub-heavy graphs of thousands of variables leave them. There
// nearly all of a skeleton's tests are run, and nearly all of those keep their edge.
//
// Both levels put a quick filter in front of the test of citest.cuh. A test keeps its edge
// for certain when |r| > thr with thr = r_c + margin_r + 8 ke / kQuickCond and the test's
// smallest pivot is at least kQuickCond (the re-test band is then no wider than that). With
// r = num / sqrt(ax ay) this is num^2 - thr^2 ax ay > 0: multiplications only, no division,
// no square root, four to five FMAs a test and (packed FP32 pairs) fewer instructions than
// that. Whatever does not pass -- a removal, a test inside the band, an ill-conditioned one --
// is evaluated by the arithmetic of citest.cuh, which alone removes edges and queues
// re-tests; so the filter only ever saves work. It is read by the warp as one vote over
// hundreds of tests.
//
// The entries come in coalesced runs, not by gathers: at level 1 from the rows of the FP32
// matrix over all p variables (wide rows hold a large part of them; the others cost their
// share of the filter and are masked after it), at level 2 from a copy of the row's
// correlation block in scratch memory.
#pragma once
#include "citest.cuh"

namespace hpc {
namespace {

// The smallest pivot the filter accepts. Smaller lets fewer ill-conditioned tests fail the
// filter but widens its band above r_c (8 ke / kQuickCond, relative to r_c 5 % at 1/32 and 1.3 %
// at 1/8 for n = 3000): edges about to be removed have many tests within it.
constexpr float kQuickCond = 1.0f / 8.0f;
constexpr float kQuickTrigger = 1e30f;  // stands for thr^2 (1 - x^2) where the test must not pass the filter

// pairs of FP32 values in 64 bits (the packed FMA of sm_100: two FMAs an instruction)
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float min3(float a, f32x2 v) {
  float x, y, d;
  unpack2(v, x, y);
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float max3(float a, f32x2 v) {
  float x, y, d;
  unpack2(v, x, y);
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(x), "f"(y));
  return d;
}

// thr^2 of the filter at a level, with slack for the filter's own roundings
__device__ __forceinline__ float quick_thr2(const Inst &I, int level) {
  const float ke = I.ke_a + (float)(level + 2) * I.ke_b;
  const float thr = (I.r_c + I.margin_r + 8.0f * ke / kQuickCond) * 1.00001f;
  return thr * thr;
}

// ---- level 1 ----------------------------------------------------------------------
//
// A test (i, j | k) and a test (j, i | k) are the same test, so an edge i < j is tested
// once, against every k of N(i) or N(j). A block takes kW1Rows rows i and L.wide_cols columns
// j > i and walks over all variables k in chunks of kW1K: the rows' entries of the chunk
// stand in shared memory, a warp loads row j's entries of the chunk into registers (32 a
// lane) and runs them against every row whose edge to j is live, so that an entry of row j
// is loaded once for up to kW1Rows edges. An edge is left at the first removal; the live
// bits carry that from chunk to chunk (no other block works on the edge).
//
// Bound: FP32 issue (a test is 4 packed half-instructions and half a three-input minimum)
// while most edges live, L2 bandwidth for the rows j of the few that stay.
constexpr int kW1K = 1024;      // variables a chunk: 32 a lane
constexpr int kW1Block = 256;  // variables between two votes
constexpr int kW1Items = kSegRows / kW1Rows;  // row groups per scan segment
static_assert(kW1Rows <= 32 && kW1K == 32 * 32, "a lane per row, a mask word per lane");
struct Wide1Smem {
  float4 x[kW1Rows][kW1K / 4];   // row entries of the chunk: lane's values v = 0..31 as 8 float4 at [v / 4 * 32 + lane]
  uint32_t mask[kW1Rows][32];    // snapshot neighbours of the rows: bit v of [lane] is variable kc + 32 v + lane
  unsigned flag[kW1Rows];             // bit q: an entry of the q-th vote block is too close to 1 for the filter
  PendRem<1> pend[kThreads / 32][kPend];
  int np[kThreads / 32];
  int next_unit;
  unsigned long long item;
};

// the test of citest.cuh at level 1: 1 remove, 0 keep, 2 undecided
__device__ __forceinline__ int test_l1(const Inst &I, float rij, float x2, float x3, float *rr_out) {
  const float ax = 1.0f - x2 * x2, ay = 1.0f - x3 * x3;
  const float cond = fminf(ax, ay);
  if (!(cond > 1e-3f)) return 2;
  const float rr = fabsf(rij - x2 * x3) * rsqrtf(ax * ay);
  *rr_out = rr;
  const float dist = rr - I.r_c;
  const float band = I.margin_r + 8.0f * __fdividef(I.ke_a + 3.0f * I.ke_b, cond);
  if (!(fabsf(dist) > band)) return 2;
  return dist < 0.0f ? 1 : 0;
}

// 32 x 32 bits across the warp: bit v of lane l becomes bit l of lane v
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x) {
  const int lane = threadIdx.x & 31;
  uint32_t m = 0x0000ffffu;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    // swap the blocks off the diagonal of every 2d x 2d block
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, d);
    x = (lane & d) ? (x & ~m) | ((y & ~m) >> d) : (x & m) | ((y & m) << d);
    m ^= m << (d >> 1);
  }
  return x;
}

// The tests of edge (i, j) in a vote block that did not pass the filter (todo: bit v for the
// lane's variable k0 + 32 v + lane), neighbours of i or j all: each by test_l1. xr: the row's
// entries of the block. True when the edge was removed. No other block works on the edge, so
// its live bits are cleared without looking. (A function of its own: inlined, its code and
// registers cost the filter loop a third of its speed.)
template <bool QO>
__device__ __noinline__ bool wide1_eval(const Launch &L, const Inst &I, int b, int i, int j, int k0, float rij,
                                        unsigned todo, const float4 *__restrict__ xr, PendRem<1> *pend, int *np,
                                        unsigned &retests) {
  const int lane = threadIdx.x & 31;
  const float *__restrict__ Cj = I.cor32 + (int64_t)j * I.p;
  unsigned undecided = 0;
  while (__any_sync(0xffffffffu, todo != 0)) {
    int res = 0, k32 = 0;
    float rr = 0.f;
    if (todo) {
      const int v = __ffs(todo) - 1;
      todo &= todo - 1;
      k32 = k0 + v * 32 + lane;
      const float x2 = reinterpret_cast<const float *>(&xr[(v >> 2) * 32 + lane])[v & 3];
      res = test_l1(I, rij, x2, __ldg(Cj + k32), &rr);
      if (res == 2) undecided |= 1u << v;
    }
    const unsigned who = __ballot_sync(0xffffffffu, res == 1);
    if (who) {
      if (lane == __ffs(who) - 1) {
        // decided in FP32: the p-value is evaluated when the records are read
        atomicAnd(I.adj + (int64_t)i * I.W + (j >> 5), ~(1u << (j & 31)));
        atomicAnd(I.adj + (int64_t)j * I.W + (i >> 5), ~(1u << (i & 31)));
        push_pending<1>(pend, np, I, b, 1, i, j, &k32, 1, -1.0 - (double)rr);
      }
      __syncwarp();
      if (*(volatile int *)np >= kPend) flush_pending<1>(L, 1, pend, np);
      return true;
    }
  }
  while (__any_sync(0xffffffffu, undecided != 0)) {
    bool rm = false;
    double pv = 0.0;
    int k32 = 0;
    if (undecided) {
      k32 = k0 + (__ffs(undecided) - 1) * 32 + lane;
      undecided &= undecided - 1;
      ++retests;
      if constexpr (QO) {
        if (!push_retest(L, b, i, j, &k32, 1)) atomicOr(&I.g->err, kErrRetestOverflow);
      } else {
        if (!(!I.cor64 && push_retest(L, b, i, j, &k32, 1))) rm = exact_remove_fast<1>(I, i, j, &k32, 1, &pv);
      }
    }
    const unsigned who = __ballot_sync(0xffffffffu, rm);
    if (who) {
      if (lane == __ffs(who) - 1 && claim_edge<false>(I, i, j)) push_pending<1>(pend, np, I, b, 1, i, j, &k32, 1, pv);
      __syncwarp();
      if (*(volatile int *)np >= kPend) flush_pending<1>(L, 1, pend, np);
      return true;
    }
  }
  return false;
}

template <bool QO>
__device__ __forceinline__ void tests_l1_wide(const Launch &L, Wide1Smem &sm) {
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  PendRem<1> *pend = sm.pend[wib];
  int *np = sm.np + wib;
  if (lane == 0) *np = 0;
  const int cols = L.wide_cols, slices = (int)((L.p_max + cols - 1) / cols);  // of the widest instance
  const unsigned long long items = (unsigned long long)L.total_segs * kW1Items * (unsigned long long)slices;
  const f32x2 minus1 = pack2(-1.f, -1.f);
  for (;;) {
    __syncthreads();
    if (tid == 0) sm.item = atomicAdd(&L.lc->tile_next, 1ull);
    __syncthreads();
    const unsigned long long item = sm.item;
    if (item >= items) break;
    const long long grp = (long long)(item / (unsigned long long)slices);
    const int jb = (int)(item - (unsigned long long)grp * (unsigned long long)slices);
    const long long seg = grp / kW1Items;
    const int b = L.count == 1 ? 0 : find_inst(L.seg_prefix, L.count, seg);
    const Inst &I = *inst_of(L, b);
    const int p = (int)I.p, W = I.W;  // p is at most 46340: variables and words are 32-bit
    const int i0 = (int)(seg - seg_begin(L, b)) * kSegRows + (int)(grp % kW1Items) * kW1Rows;
    const int j_lo = jb * cols, j_hi = min(p, j_lo + cols);
    if (i0 >= p || j_hi <= i0 + 1 || csr_overflow(I)) continue;  // no pair i < j in the item
    const int w_lo = j_lo >> 5, w_hi = (j_hi + 31) >> 5;
    const float *__restrict__ C = I.cor32;
    const float thr2 = quick_thr2(I, 1);
    const f32x2 nthr2 = pack2(-thr2, -thr2);
    unsigned executed = 0, retests = 0;
    // the live edges of row i to the columns of word w, j > i
    auto live_word = [&](int i, int w) -> uint32_t {
      const uint32_t x = *(volatile const uint32_t *)(I.adj + (int64_t)i * W + w);
      return w * 32 > i ? x : w * 32 + 31 <= i ? 0u : x & (0xfffffffeu << (i & 31));
    };
    for (int kc = 0; kc < p; kc += kW1K) {
      __syncthreads();  // the chunk before is done with, and its removals are in the live bits
      if (tid == 0) sm.next_unit = w_lo * 4;
      if (tid < kW1Rows) sm.flag[tid] = 0;
      // does any edge of the item still live? (the last chunks of most items are empty)
      bool any = false;
      for (int t = tid; t < kW1Rows * (w_hi - w_lo); t += kThreads) {
        const int i = i0 + t % kW1Rows;
        if (i < p) any |= live_word(i, w_lo + t / kW1Rows) != 0;
      }
      if (!__syncthreads_or(any)) break;
      for (int t = tid; t < kW1Rows * (kW1K / 4); t += kThreads) {
        const int r = t / (kW1K / 4), q = t % (kW1K / 4), v4 = q >> 5;  // q & 31: the lane that will read it
        const int i = i0 + r, k = kc + v4 * 128 + (q & 31);
        const float *__restrict__ Ci = C + (int64_t)i * p;
        float x[4];
        bool close = false;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          x[u] = (i < p && k + 32 * u < p && k + 32 * u != i) ? __ldg(Ci + k + 32 * u) : 0.f;
          close |= 1.0f - x[u] * x[u] < kQuickCond;
        }
        sm.x[r][q] = make_float4(x[0], x[1], x[2], x[3]);
        if (close) atomicOr(&sm.flag[r], 1u << (v4 / (kW1Block / 128)));
      }
      const int gw = (kc >> 5) + lane;  // the lane's mask word of the chunk
      for (int r = wib; r < kW1Rows; r += kThreads / 32)
        sm.mask[r][lane] = warp_transpose((i0 + r < p && gw < W) ? __ldcg(I.adj0 + (int64_t)(i0 + r) * W + gw) : 0u);
      __syncthreads();
      const int blocks = min(kW1K / kW1Block, (p - kc + kW1Block - 1) / kW1Block);
      for (;;) {  // 8 columns j at a time, as the warps come
        int w = 0;
        if (lane == 0) w = atomicAdd(&sm.next_unit, 1);
        w = __shfl_sync(0xffffffffu, w, 0);
        if (w >= w_hi * 4) break;
        const uint32_t byte = 0xffu << ((w & 3) * 8);
        w >>= 2;
        const uint32_t word = (lane < kW1Rows && i0 + lane < p) ? live_word(i0 + lane, w) & byte : 0u;  // lane: row
        unsigned todo_j = __reduce_or_sync(0xffffffffu, word);
        while (todo_j) {
          const int q = __ffs(todo_j) - 1;
          todo_j &= todo_j - 1;
          const int j = w * 32 + q;
          unsigned rows = __ballot_sync(0xffffffffu, (word >> q) & 1u);
          const float *__restrict__ Cj = C + (int64_t)j * p + kc + lane;
          float rij_l = 0.f;
          if ((word >> q) & 1u) rij_l = __ldg(C + (int64_t)(i0 + lane) * p + j);
          const uint32_t mw = gw < W ? __ldcg(I.adj0 + (int64_t)j * W + gw) : 0u;
          f32x2 xj[16], ay[16];  // r_jk and thr^2 (1 - r_jk^2), the lane's variables kc + 32 v + lane
          {
            float x[32];
            if (kc + kW1K <= p) {
#pragma unroll
              for (int v = 0; v < 32; ++v) x[v] = __ldg(Cj + 32 * v);
            } else {
#pragma unroll
              for (int v = 0; v < 32; ++v) x[v] = kc + 32 * v + lane < p ? __ldg(Cj + 32 * v) : 0.f;
            }
            const bool own = (unsigned)(j - kc) < (unsigned)kW1K;  // j itself in the chunk
            if (own) {
#pragma unroll
              for (int v = 0; v < 32; ++v)
                if (kc + 32 * v + lane == j) x[v] = 0.f;
            }
            float worst = -1.f;
#pragma unroll
            for (int v = 0; v < 16; ++v) {
              xj[v] = pack2(x[2 * v], x[2 * v + 1]);
              const f32x2 na = fma2(xj[v], xj[v], minus1);  // -(1 - r_jk^2)
              ay[v] = mul2(na, nthr2);
              worst = max3(worst, na);
            }
            // an entry too close to 1 for the filter: its tests must not pass (rare)
            if (__any_sync(0xffffffffu, worst > -kQuickCond)) {
#pragma unroll
              for (int v = 0; v < 16; ++v) {
                const float y0 = 1.0f - x[2 * v] * x[2 * v], y1 = 1.0f - x[2 * v + 1] * x[2 * v + 1];
                ay[v] = pack2(y0 < kQuickCond ? kQuickTrigger : thr2 * y0, y1 < kQuickCond ? kQuickTrigger : thr2 * y1);
              }
            }
          }
          const uint32_t mj = warp_transpose(mw);  // bit v: kc + 32 v + lane is a snapshot neighbour of j
          while (rows) {
            const int r = __ffs(rows) - 1;
            rows &= rows - 1;
            const int i = i0 + r;
            const float rij = __shfl_sync(0xffffffffu, rij_l, r);
            const f32x2 nrij = pack2(-rij, -rij);
            const unsigned flag = sm.flag[r];
            const float4 *__restrict__ xr = sm.x[r];
            // the tests of the chunk: neighbours of i or j, without i and j
            uint32_t nb = sm.mask[r][lane] | mj;
            if ((unsigned)(i - kc) < (unsigned)kW1K && (i & 31) == lane) nb &= ~(1u << ((i - kc) >> 5));
            if ((unsigned)(j - kc) < (unsigned)kW1K && (j & 31) == lane) nb &= ~(1u << ((j - kc) >> 5));
            bool gone = false;
#pragma unroll
            for (int blk = 0; blk < kW1K / kW1Block; ++blk) {
              if (blk < blocks && !gone) {
                float low = 0.f;
#pragma unroll
                for (int v4 = blk * (kW1Block / 128); v4 < (blk + 1) * (kW1Block / 128); ++v4) {
                  const float4 xv = xr[v4 * 32 + lane];
                  const f32x2 xa = pack2(xv.x, xv.y), xb = pack2(xv.z, xv.w);
                  // num = r_ik r_jk - r_ij; num^2 - thr^2 (1 - r_ik^2) (1 - r_jk^2)
                  const f32x2 na = fma2(xa, xj[2 * v4], nrij), nb2 = fma2(xb, xj[2 * v4 + 1], nrij);
                  const f32x2 ta = mul2(fma2(xa, xa, minus1), ay[2 * v4]);
                  const f32x2 tb = mul2(fma2(xb, xb, minus1), ay[2 * v4 + 1]);
                  low = min3(low, fma2(na, na, ta));
                  low = min3(low, fma2(nb2, nb2, tb));
                }
                const uint32_t nbb = (nb >> (blk * (kW1Block / 32))) & ((1u << (kW1Block / 32)) - 1u);
                executed += (unsigned)__popc(nbb);
                const bool all = (flag >> blk) & 1u;
                if (__any_sync(0xffffffffu, low < 0.f) || all) {
                  unsigned todo = all ? nbb : 0u;  // which of the lane's tests did not pass
                  if (!all && low < 0.f) {
#pragma unroll
                    for (int v4 = 0; v4 < kW1Block / 128; ++v4) {
                      const float4 xv = xr[(blk * (kW1Block / 128) + v4) * 32 + lane];
#pragma unroll
                      for (int h = 0; h < 2; ++h) {
                        const int at = 2 * (blk * (kW1Block / 128) + v4) + h;
                        const f32x2 x2 = h ? pack2(xv.z, xv.w) : pack2(xv.x, xv.y);
                        const f32x2 n2 = fma2(x2, xj[at], nrij);
                        float s0, s1;
                        unpack2(fma2(n2, n2, mul2(fma2(x2, x2, minus1), ay[at])), s0, s1);
                        if (s0 < 0.f) todo |= 1u << (4 * v4 + 2 * h);
                        if (s1 < 0.f) todo |= 2u << (4 * v4 + 2 * h);
                      }
                    }
                    todo &= nbb;
                  }
                  if (__any_sync(0xffffffffu, todo != 0))
                    gone = wide1_eval<QO>(L, I, b, i, j, kc + blk * kW1Block, rij, todo, xr + blk * (kW1Block / 4),
                                          pend, np, retests);
                }
              }
            }
          }
        }
      }
    }
    const unsigned ex = __reduce_add_sync(0xffffffffu, executed), rt = __reduce_add_sync(0xffffffffu, retests);
    if (lane == 0) {
      if (ex) atomicAdd(&I.ctr[1].tests, (unsigned long long)ex);
      if (rt) atomicAdd(&I.ctr[1].retests, (unsigned long long)rt);
    }
  }
  __syncwarp();
  flush_pending<1>(L, 1, pend, np);
}

// ---- level 2 ----------------------------------------------------------------------
//
// Given the first member a, level 2 is level 1 on the correlations conditioned on a: with
// R_x = r_ax, G_x = 1 / sqrt(1 - R_x^2) and U_x = (r_ix - r_ia R_x) G_x / sqrt(1 - r_ia^2), the
// test (i, j | a, b) is
//   num = U'_j - U_b w,  w = (r_jb - R_j R_b) G_b,  U'_j = (r_ij - r_ia R_j) / sqrt(1 - r_ia^2),
//   r^2 = num^2 / ((1 - U_b^2) e),  e = (1 - R_j^2) - w^2,
// five FMAs a test once R, G and U of the b's are formed -- which is done once for kW2A members
// a and 128 members b (four a lane) and serves every live j of the warp. A block takes a wide
// row i (or up to wide2_slice of its neighbours j, where there are more) and copies the row's
// correlation block -- row i and the slice's rows over {i} and N(i), block-local indices as in
// stage_block -- into its scratch, so that all these loads are coalesced. The members a go by
// in steps of kW2Super, kW2A of them to each warp, which runs them against every live j of the
// slice: forming R, G and U takes as long as several j's tests, so it has to serve many, and most
// edges of a wide row are removed after a few steps. The warps go round the j's from different
// places, so that a j that one of them removes is not tested by those that come to it later. The
// live bits (other rows remove edges too) are read again every step.
//
// Bound: FP32 issue while many edges live (3.5 instructions a test), the copy of the block
// (one gather an entry) where few do.
constexpr int kW2A = 4;         // members a at a time
constexpr int kW2Chunk = 128;   // members b at a time: four a lane
static_assert(kW2Super == kW2A * (kThreads / 32), "a warp per kW2A members of a step");
static_assert(kW2Slice % kThreads == 0 && kW2Slice / kThreads <= 32, "a thread watches kW2Slice / kThreads members");

constexpr int kW2Ahead = 4;     // rows j in flight to a warp's ring
struct Wide2Smem {
  float4 ring[kThreads / 32][kW2Ahead][32];  // rows j of the chunk, a lane's four b's each
  // per j of the warp's 32 and a: R_j, U'_j, -(1 - R_j^2) and, for the first a, the j's tests in the chunk
  float4 s[kThreads / 32][32][kW2A];
};
struct Wide2Lists {
  unsigned alive[kW2Slice / 32];  // the listed j's still live in this step
  uint16_t list[kW2Slice];        // the slice members alive at the step's start
  int total;
  unsigned item;
  unsigned long long executed;    // the item's tests
};

// The tests of edge (i, j), j = neighbour xj - 1 of the row, with first members xa0 .. xa0 +
// kW2A - 1 and second members x0 .. x0 + kW2Chunk - 1 (block-local) that did not pass the
// filter (todo: bit 4 a + u for first member xa0 + a and the lane's second member x0 + 4 lane +
// u): each by test_f32_inc on the copied block. ri, rj and ra0 + a * ld: the rows of i, j and the
// first members (written by this kernel: no read-only loads). True when the edge was removed.
__device__ __noinline__ bool wide2_eval(const Launch &L, const Inst &I, int b, int64_t i, int base, int d, int xj,
                                        int xa0, int x0, unsigned todo, const float *ri, const float *rj,
                                        const float *ra0, int64_t ld, PendRem<2> *pend, int *np, unsigned &retests) {
  const int lane = threadIdx.x & 31;
  const int64_t j = I.colidx[base + xj - 1];
  unsigned undecided = 0;
  for (int pass = 0; pass < 2; ++pass) {  // the tests in FP32, then those left undecided
    unsigned &bits = pass == 0 ? todo : undecided;
    while (__any_sync(0xffffffffu, bits != 0)) {
      bool rm = false;
      double pv = 0.0;
      int ids[2] = {0, 0};
      if (bits) {
        const int t = __ffs(bits) - 1;
        bits &= bits - 1;
        const int xa = xa0 + (t >> 2), xb = x0 + lane * 4 + (t & 3);
        if (xa < d && xb > xa && xb <= d && xa != xj && xb != xj) {
          ids[0] = I.colidx[base + xa - 1];
          ids[1] = I.colidx[base + xb - 1];
          if (pass == 0) {
            // the five entries as the 4 x 4 block of (i, j, a, b)
            const float m[16] = {0.f, ri[xj], ri[xa], ri[xb], 0.f, 0.f, rj[xa], rj[xb],
                                 0.f, 0.f, 0.f, ra0[(int64_t)(t >> 2) * ld + xb], 0.f, 0.f, 0.f, 0.f};
            const int xs[2] = {2, 3};
            Fact<2> F;
            float rr = 0.f;
            const int res = test_f32_inc<2>(I, m, 4, 0, 1, xs, 2, 0, F, &rr);
            rm = res == 1;
            pv = -1.0 - (double)rr;  // decided in FP32: the p-value is evaluated when the records are read
            if (res == 2) undecided |= 1u << t;
          } else {
            ++retests;
            if (!(!I.cor64 && push_retest(L, b, i, j, ids, 2))) rm = exact_remove_fast<2>(I, i, j, ids, 2, &pv);
          }
        }
      }
      const unsigned who = __ballot_sync(0xffffffffu, rm);
      if (who) {
        // another row's test may have removed the edge meanwhile
        if (lane == __ffs(who) - 1 && claim_edge(I, i, j)) push_pending<2>(pend, np, I, b, 2, i, j, ids, 2, pv);
        __syncwarp();
        if (*(volatile int *)np >= kPend) flush_pending<2>(L, 2, pend, np);
        return true;
      }
    }
  }
  return false;
}

// rows of the block copied by the whole thread block: row q of dst = the row of neighbour
// x_first + q (block-local index) over {i} and N(i), zero on its own position; x_first = 0: row i
__device__ __forceinline__ void wide2_copy(const Inst &I, int64_t i, int base, int d, int64_t ld, int x_first,
                                           int step, int rows, float *dst) {
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  for (int q = wib; q < rows; q += kThreads / 32) {
    const int x = x_first + q * step;
    const int64_t v = x == 0 ? i : (int64_t)I.colidx[base + x - 1];
    const float *__restrict__ Cv = I.cor32 + v * I.p;
    float *out = dst + (int64_t)q * ld;
#pragma unroll 4
    for (int y = lane; y < (int)ld; y += 32) {
      const int64_t c = y == 0 ? i : y <= d ? (int64_t)I.colidx[base + y - 1] : v;
      out[y] = (y > d || y == x) ? 0.f : __ldg(Cv + c);
    }
  }
}

__device__ __forceinline__ void tests_l2_wide(const Launch &L, Wide2Smem &sm, PendRem<2> *pend_all, int *np_all) {
  __shared__ Wide2Lists ls;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  constexpr int kWarps = kThreads / 32;
  PendRem<2> *pend = pend_all + wib * kPend;
  int *np = np_all + wib;
  if (lane == 0) *np = 0;
  __syncthreads();
  const unsigned int n_front = *(volatile unsigned int *)&L.lc->wide_front;
  const unsigned int n_back = *(volatile unsigned int *)&L.lc->wide_back;
  float *scratch = L.wide_scratch + (int64_t)blockIdx.x * L.wide_floats;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      ls.item = atomicAdd(&L.lc->wide_next, 1u);
      ls.executed = 0;
    }
    __syncthreads();
    const unsigned item = ls.item;
    if (item >= n_front + n_back) break;
    // the widest rows come first: they take longest
    const WideItem it = L.wide_items[item < n_front ? item : L.wide_cap - 1 - (item - n_front)];
    const Inst &I = *inst_of(L, it.inst);
    const int b = it.inst;
    const int64_t i = it.row;
    const int d = I.deg[i], base = I.rowptr[i];
    const int ns = wide2_slices(d, I.p);
    const int64_t ld = wide2_ld(d);
    const int m = (d - it.slice + ns - 1) / ns;  // the slice's neighbours: it.slice, it.slice + ns, ...
    float *ri = scratch, *rows = scratch + ld, *arows = rows + (int64_t)min(d, wide2_slice(d, I.p)) * ld;
    wide2_copy(I, i, base, d, ld, 0, 1, 1, ri);
    wide2_copy(I, i, base, d, ld, 1 + it.slice, ns, m, rows);
    const float thr2 = quick_thr2(I, 2);
    unsigned retests = 0;
    unsigned gone = 0;  // bit w: slice member tid + kThreads w is known to be removed
    for (int xs0 = 1; xs0 < d; xs0 += kW2Super) {
      // the slice's live members
      __syncthreads();  // the step before is done with the rows a and the list
      if (tid == 0) ls.total = 0;
      __syncthreads();
      for (int w = 0; w * kThreads < m; ++w) {
        const int t = tid + w * kThreads;
        bool on = t < m && !((gone >> w) & 1u);
        if (on) on = live_bit(I.adj, I.W, i, I.colidx[base + it.slice + t * ns]);
        if (!on) gone |= 1u << w;
        const unsigned mask = __ballot_sync(0xffffffffu, on);
        int at = 0;
        if (lane == 0 && mask) at = atomicAdd(&ls.total, __popc(mask));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (on) ls.list[at + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)t;
      }
      __syncthreads();
      const int total = ls.total;
      if (total == 0) break;
      if (tid < kW2Slice / 32) {
        const int n = min(32, max(0, total - 32 * tid));
        ls.alive[tid] = n == 32 ? ~0u : (1u << n) - 1u;
      }
      if (ns > 1) wide2_copy(I, i, base, d, ld, xs0, 1, min(kW2Super, d + 1 - xs0), arows);
      __syncthreads();
      const int groups = (total + 31) >> 5;
      const int xa0 = xs0 + wib * kW2A;  // the warp's members a of the step
      if (xa0 >= d) continue;
      const float *ra0 = ns == 1 ? rows + (int64_t)(xa0 - 1) * ld : arows + (int64_t)(xa0 - xs0) * ld;
      float ria[kW2A], inv_i[kW2A];
#pragma unroll
      for (int a = 0; a < kW2A; ++a) {
        ria[a] = xa0 + a < d ? ri[xa0 + a] : 0.f;
        inv_i[a] = rsqrtf(fmaxf(1.0f - ria[a] * ria[a], 1e-6f));
      }
      unsigned executed = 0;  // the lane's j's tests with the step's members a
      for (int x0 = (xa0 + 1) / kW2Chunk * kW2Chunk; x0 <= d; x0 += kW2Chunk) {
        const int xb = x0 + lane * 4;
        const bool load = xb < (int)ld;
        // G_b, R_b G_b, U_b and thr^2 (1 - U_b^2) of the lane's four b's for each a
        f32x2 G[kW2A][2], RG[kW2A][2], U[kW2A][2], TU[kW2A][2];
        {
          const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 vi = load ? *reinterpret_cast<const float4 *>(ri + xb) : zero;
          const float rib[4] = {vi.x, vi.y, vi.z, vi.w};
#pragma unroll
          for (int a = 0; a < kW2A; ++a) {
            const bool on = xa0 + a < d;
            const float4 va = load && on ? *reinterpret_cast<const float4 *>(ra0 + (int64_t)a * ld + xb) : zero;
            const float R[4] = {va.x, va.y, va.z, va.w};
            float g[4], rg[4], uu[4], tu[4];
            const float ai = 1.0f - ria[a] * ria[a];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const bool in = xb + u > xa0 + a && xb + u <= d && on;
              const float q = 1.0f - R[u] * R[u];
              const float gg = rsqrtf(fmaxf(q, 1e-6f));
              const float un = (rib[u] - ria[a] * R[u]) * gg * inv_i[a];
              const float au = 1.0f - un * un;
              // a pivot too small for the filter: the test must not pass
              const bool bad = !(q >= kQuickCond && ai * au >= kQuickCond);
              g[u] = in ? gg : 0.f;
              rg[u] = in ? R[u] * gg : 0.f;
              uu[u] = in ? un : 0.f;
              tu[u] = !in ? -1.f : bad ? kQuickTrigger : thr2 * au;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              G[a][h] = pack2(g[2 * h], g[2 * h + 1]);
              RG[a][h] = pack2(rg[2 * h], rg[2 * h + 1]);
              U[a][h] = pack2(uu[2 * h], uu[2 * h + 1]);
              TU[a][h] = pack2(tu[2 * h], tu[2 * h + 1]);
            }
          }
        }
        for (int gi = 0; gi < groups; ++gi) {  // 32 of the j's at a time, each warp from its own place on
          const int grp = (gi + wib) % groups;
          const unsigned alive = __shfl_sync(0xffffffffu, *(volatile unsigned *)&ls.alive[grp], 0);
          if (!alive) continue;
          const bool mine = (alive >> lane) & 1u;
          const int t_l = mine ? ls.list[grp * 32 + lane] : 0;
          // the j's in turn, from a place of the warp's own; their rows come kW2Ahead ahead
          const int turn = wib * 4;
          unsigned fetch = __funnelshift_r(alive, alive, turn), left = fetch;
          int slot_in = 0, slot = 0;
          auto request = [&]() {
            const int q = fetch ? (__ffs(fetch) - 1 + turn) & 31 : 0;
            const int t = __shfl_sync(0xffffffffu, t_l, q);
            if (fetch && load) {
              const uint32_t to = (uint32_t)__cvta_generic_to_shared(&sm.ring[wib][slot_in][lane]);
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(rows + (int64_t)t * ld + xb)
                           : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            fetch &= fetch - 1;
            slot_in = (slot_in + 1) & (kW2Ahead - 1);
          };
#pragma unroll
          for (int k = 0; k < kW2Ahead - 1; ++k) request();
          // the lane's j: R_j, U'_j and -(1 - R_j^2) for the members a, and its tests here (all second
          // members of the chunk, for each a, but j itself), taken off again where they are not run
          if (mine) {
            const int xj = 1 + it.slice + t_l * ns;  // block-local
            const float rij = ri[xj];
            int cnt = 0;
#pragma unroll
            for (int a = 0; a < kW2A; ++a) {
              const int xa = xa0 + a, lo = max(xa + 1, x0), hi = min(x0 + kW2Chunk - 1, d);
              const float R = xa < d ? ra0[(int64_t)a * ld + xj] : 0.f;
              sm.s[wib][lane][a] = make_float4(R, (rij - ria[a] * R) * inv_i[a], R * R - 1.0f, 0.f);
              if (xa < d && xa != xj && hi >= lo) cnt += hi - lo + 1 - (xj >= lo && xj <= hi ? 1 : 0);
            }
            sm.s[wib][lane][0].w = __int_as_float(cnt);
            executed += (unsigned)cnt;
          }
          __syncwarp();
          while (left) {
            const int q = (__ffs(left) - 1 + turn) & 31;
            left &= left - 1;
            request();
            asm volatile("cp.async.wait_group %0;" ::"n"(kW2Ahead - 1) : "memory");
            const float4 v = sm.ring[wib][slot][lane];  // the lane's own copy
            slot = (slot + 1) & (kW2Ahead - 1);
            // removed by another warp meanwhile?
            if (!((__shfl_sync(0xffffffffu, *(volatile unsigned *)&ls.alive[grp], 0) >> q) & 1u)) {
              if (lane == q) executed -= (unsigned)__float_as_int(sm.s[wib][lane][0].w);
              continue;
            }
            const f32x2 r01 = pack2(-v.x, -v.y), r23 = pack2(-v.z, -v.w);  // -r_jb
            float low = 0.f, high = -1.f;
#pragma unroll
            for (int a = 0; a < kW2A; ++a) {
              const float4 sc = sm.s[wib][q][a];
              const f32x2 R2 = pack2(sc.x, sc.x), U2 = pack2(sc.y, sc.y), q2 = pack2(sc.z, sc.z);
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const f32x2 wn = fma2(R2, RG[a][h], mul2(h ? r23 : r01, G[a][h]));  // -w
                const f32x2 num = fma2(U[a][h], wn, U2);
                const f32x2 en = fma2(wn, wn, q2);  // -e
                low = min3(low, fma2(num, num, mul2(TU[a][h], en)));
                high = max3(high, en);
              }
            }
            if (!__any_sync(0xffffffffu, low < 0.f || high > -kQuickCond)) continue;
            unsigned todo = 0;  // which of the lane's tests did not pass
            if (low < 0.f || high > -kQuickCond) {
#pragma unroll
              for (int a = 0; a < kW2A; ++a) {
                const float4 sc = sm.s[wib][q][a];
                const f32x2 R2 = pack2(sc.x, sc.x), U2 = pack2(sc.y, sc.y), q2 = pack2(sc.z, sc.z);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const f32x2 wn = fma2(R2, RG[a][h], mul2(h ? r23 : r01, G[a][h]));
                  const f32x2 num = fma2(U[a][h], wn, U2);
                  const f32x2 en = fma2(wn, wn, q2);
                  float s0, s1, e0, e1;
                  unpack2(fma2(num, num, mul2(TU[a][h], en)), s0, s1);
                  unpack2(en, e0, e1);
                  if (s0 < 0.f || e0 > -kQuickCond) todo |= 1u << (4 * a + 2 * h);
                  if (s1 < 0.f || e1 > -kQuickCond) todo |= 2u << (4 * a + 2 * h);
                }
              }
            }
            const int t = __shfl_sync(0xffffffffu, t_l, q);
            if (wide2_eval(L, I, b, i, base, d, 1 + it.slice + t * ns, xa0, x0, todo, ri, rows + (int64_t)t * ld, ra0,
                           ld, pend, np, retests)) {
              if (lane == 0) atomicAnd(&ls.alive[grp], ~(1u << q));
            }
          }
          asm volatile("cp.async.wait_group 0;" ::: "memory");  // the ring is free for the next group
          __syncwarp();                                          // ... and so are the scalars
        }
      }
      executed = __reduce_add_sync(0xffffffffu, executed);
      if (lane == 0) atomicAdd(&ls.executed, (unsigned long long)executed);
    }
    const unsigned rt = __reduce_add_sync(0xffffffffu, retests);
    if (lane == 0 && rt) atomicAdd(&I.ctr[2].retests, (unsigned long long)rt);
    __syncthreads();
    if (tid == 0 && ls.executed) atomicAdd(&I.ctr[2].tests, ls.executed);
  }
  __syncwarp();
  flush_pending<2>(L, 2, pend, np);
}

}  // namespace
}  // namespace hpc
