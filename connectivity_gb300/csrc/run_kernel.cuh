// k_run: a whole run (trim, reachability, colour rounds) in one cooperative
// launch, and its launch helpers.
#pragma once
#include "run_device.cuh"
#include "residual_device.cuh"

namespace gb {
namespace {

// Device time at a phase boundary (block 0, thread 0), into the run's slot
// of the context's phase-time ring.
__device__ __forceinline__ void phase_mark(const Args& A, int i) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.w.tphase != nullptr) A.w.tphase[i] = gtimer();
}

// ------------------------------------------------------------------------
// k_run: one run (trim, reachability, colour rounds) in one cooperative
// launch; a grid barrier separates the phases, so each phase sees the
// previous one's lists, counters and pivot.  NC: adjacency lists walked by
// the reachability phase (1, or 2 for WCC of a directed graph).
// ------------------------------------------------------------------------
// kOptions: the optional features are compiled in: FW-BW rounds after the
// first, each from a new pivot while at least kRepivotMin vertices are valid
// (fwbw_rounds > 1, single graphs), and the edge-balanced push
// (expand_mode 1).  That variant is compiled in its own translation unit
// (kernels_options.cu), so the code of the default run is the same with or
// without it.
// Extra: a phase between the trim and the searches (NoExtra, or the
// contraction of kernels_contract.cu), likewise in a unit of its own.
struct NoExtra {
  static constexpr bool kOn = false;
};
template <int NC, bool kOptions, class Extra = NoExtra>
__global__ void __launch_bounds__(kBlock, kMinBlocks) k_run(Args A) {
  __shared__ Smem sm;
  sm.stage_base = g_dyn_smem;
  bar_open();
  Ctl* c = A.w.ctl;
  phase_mark(A, 0);
  trim_phase(A, sm);
  if (!grid_barrier(c, 900)) return;
  phase_mark(A, 1);
  if constexpr (Extra::kOn) {
    Extra::run(A, sm);
    if (!grid_barrier(c, 904)) return;
  }
  reach_phase<NC, false, kOptions>(A, sm);
  if constexpr (kOptions) {
    for (int r = 1; r < A.p.fwbw_rounds && A.g.batch.gid == nullptr; ++r) {
      if (!grid_barrier(c, 32)) return;  // the last round's valid count
      if (__ldcg(&c->nvalid) < kRepivotMin) break;
      if (!repivot(A, sm)) return;
      if (__ldcg(&c->rpivot) < 0) break;
      reach_phase<NC, true, true>(A, sm);
    }
  }
  if (!grid_barrier(c, 901)) return;
  phase_mark(A, 2);
  // (every block reads the same counts after a barrier, so all take the
  // same branches)
  const bool scc = A.kind == kSCC;
  bool left = true;
  if constexpr (NC == 1) {
    if (scc && A.p.colour_mode == 2 && A.p.free_steps) {
      left = residual_phase(A, sm);
      if (left && !grid_barrier(c, 905)) return;
    }
  }
  if (left && scc &&
      (A.p.colour_mode == 1 || (A.p.colour_mode == 2 && __ldcg(&c->nvalid) >= kSigMin))) {
    signature_rounds(A, sm, A.w.listA, A.w.listB);
  } else if (left) {
    // colour_mode 2: a residual still left after kSigAfter colour rounds
    // goes on in signature rounds (a deep condensation: chains)
    const int cap = scc && A.p.colour_mode == 2 ? kSigAfter : 0x7fffffff;
    int32_t* cur = A.w.listA;
    if (scc || A.g.in.off == nullptr) colour_rounds<1>(A, sm, cap, &cur);
    else colour_rounds<2>(A, sm, cap, &cur);
    if (cap != 0x7fffffff) {
      if (!grid_barrier(c, 903)) return;
      if (__ldcg(&c->nvalid) > 0 && !ld_vol(&c->err))
        signature_rounds(A, sm, cur, cur == A.w.listA ? A.w.listB : A.w.listA);
    }
  }
  if (!grid_barrier(c, 902)) return;
  phase_mark(A, 3);
}

template <class K>
cudaError_t coop(K kern, int grid, const Args& a, cudaStream_t s) {
  void* params[] = {const_cast<Args*>(&a)};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(grid), dim3(kBlock), params,
                                     (size_t)kDynSmem, s);
}

// Blocks per SM of a run kernel at kDynSmem bytes of dynamic shared memory
// (0 on an error).
template <class K>
int run_blocks_per_sm(K kern) {
  if (cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kDynSmem) != cudaSuccess)
    return 0;
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)kern, kBlock, kDynSmem) !=
      cudaSuccess)
    return 0;
  return per;
}

}  // namespace
}  // namespace gb
