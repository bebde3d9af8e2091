// The level kernel: the phases of one level l >= 1 in one cooperative launch.
#pragma once
#include "citest.cuh"
#include "wide.cuh"

namespace hpc {
namespace {

// One level l >= 1: rebuild | grid barrier | scan | grid barrier | CI tests. LT = 1
// is the lane-interleaved level-1 body (V: kL1Prefetch loads one step ahead,
// kL1Chunked runs the chunked body of the higher levels; picked by the tile policy),
// LT = 2..16 the bodies unrolled for l = LT (V = kSetOrder: in the set order, LT up to
// kSetTop), LT = 0 the runtime-level body; V = kWide: the wide-row bodies of levels 1 and 2.
constexpr int variant_blocks(int lt, int v, int set_blocks) {  // resident blocks per SM
  return v == kSetOrder ? set_blocks : (lt == 1 && !(v & kWide) && (v & 3) != kL1Chunked) ? 4 : 2;
}
template <int LT, bool MIXED, int V = kL1Interleaved>
__global__ void __launch_bounds__(kThreads, variant_blocks(LT, V, kSetBlocks<LT>))
    level_kernel(const __grid_constant__ Launch L) {
  // the row offsets of own_scan, or the wide bodies' chunk and ring
  extern __shared__ __align__(16) unsigned long long rw_smem[];
  constexpr int kUnits = V == kSetOrder ? kUnitSets : (LT == 2 && V == kWide) ? kUnitNarrow : kUnitTests;
  unsigned int epoch = 0;
  const bool stamp = blockIdx.x == 0 && threadIdx.x == 0;  // the phase times
  if (stamp) L.lc->t_entry = globaltimer_ns();
  rebuild_phase(L, kUnits, LT == 1 && (V & kWide) != 0);
  if (!grid_barrier(L, epoch)) return;
  if (stamp) L.lc->t_rebuilt = globaltimer_ns();
  // (level 1 leaves its shared memory to the L1 cache, the wide-row kernels need the queue of the scan)
  constexpr bool kOwn = LT != 1 && (V == kSetOrder || !(V & kWide));
  int max_deg = 0;
  Work wk{0, nullptr, L.work_prefix, L.count};
  if (kOwn && L.row_cache) {
    wk.total = own_scan(L, kUnits, rw_smem, &max_deg);
    wk.own = rw_smem;
  } else {
    scan_phase(L, kUnits);
    if (!grid_barrier(L, epoch)) return;
    wk.total = L.work_prefix[L.count];
    max_deg = *(volatile const int *)&L.lc->max_deg;
  }
  if (stamp) L.lc->t_scanned = globaltimer_ns();
  const TuneEntry te = tile_policy(L, max_deg);
  if constexpr (V == kSetOrder) {
    static_assert(MIXED && LT >= 2 && LT <= kSetTop, "the set order runs levels 2-24 in mixed precision");
    __shared__ TestSmem<LT, true> sm;
    tests_set<LT>(L, wk, te, sm);
  } else if constexpr (LT == 1 && (V & kWide) != 0) {
    static_assert(MIXED, "the wide-row kernels run in mixed precision");
    tests_l1_wide<(V & kQueueOnly) != 0>(L, *reinterpret_cast<Wide1Smem *>(rw_smem));
  } else if constexpr (LT == 2 && V == kWide) {
    __shared__ TestSmem<2, true> sm;
    static_assert(sizeof(Wide2Smem) <= sizeof(sm.blk), "the wide rows' scalars stand where the staged blocks do");
    tests_l2_wide(L, *reinterpret_cast<Wide2Smem *>(sm.blk), sm.pend[0], sm.np);
    __syncthreads();
    tests_generic<2, true>(L, wk, te, sm);
  } else if constexpr (LT == 1 && (V & 3) != kL1Chunked) {  // level 1 keeps the SM's on-chip memory for L1 cache
    tests_l1<MIXED, (V & 3) == kL1Prefetch, (V & kQueueOnly) != 0>(L, wk, te);
  } else {
    __shared__ TestSmem<LT, MIXED> sm;
    tests_generic<LT, MIXED>(L, wk, te, sm);
  }
  if (kOwn && wk.own && blockIdx.x == gridDim.x - 1 && threadIdx.x < 32) {
    __syncwarp();
    own_summary(L, wk.total, max_deg);
  }
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(&L.lc->t_end, globaltimer_ns());
}

}  // namespace
}  // namespace hpc
