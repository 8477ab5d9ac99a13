// jsh_forms.cu -- the mixed path's other forms: the static schedule (one item
// per thread to completion) and the single-kernel persistent schedule (both
// passes in one kernel).  Compiled twice, like jsh_persistent.cu:
// jsh_forms_ft.cu builds it with the Faraday-thick mode.
#include "jsh_mixed.cuh"

#include "jsh_split.h"

namespace jsh {

namespace {

// One thread per work item, stepped to completion.
template <bool FULL>
__global__ void __launch_bounds__(128) transfer_static_mixed_kernel(const JshRequest* __restrict__ reqs,
                                                                     int n_req) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  extern __shared__ float ksh[];
  batch_prefix(reqs, n_req, base);
  const unsigned long long w = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  float* K = ksh + threadIdx.x * form_words<FULL>();
  Tally T = tally_new();
  if (w < base[n_req]) {
    Lane L;
    lane_start<PASS_BOTH>(L, reqs, base, n_req, w, false);
    while (L.phase != PH_IDLE) lane_advance<FULL, PASS_BOTH>(L, reqs, K, T);
  }
  tally_flush(T, reqs);
}

// Persistent CTAs: each warp keeps 32 lanes busy, refilling idle lanes from
// the global queue when at least `refill` of them are idle.  COMPACT builds
// the kernel for at most 128 threads and 3 resident CTAs per SM, which caps
// it at 168 registers (no spills) instead of 182: 12 instead of 10
// resident warps per SM, more latency hiding for the bulk of short rays at
// the price of issue slots for the long ones; the autotuner picks.
template <bool FULL, bool COMPACT>
__global__ void __launch_bounds__(COMPACT ? 128 : 256, COMPACT ? 3 : 1)
    transfer_persistent_mixed_kernel(const JshRequest* __restrict__ reqs, int n_req, unsigned long long* queue,
                                     int refill) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  extern __shared__ float ksh[];
  batch_prefix(reqs, n_req, base);
  float* K = ksh + threadIdx.x * form_words<FULL>();
  const unsigned long long total = base[n_req];
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt_mask = (1u << lane) - 1u;
  Lane L;
  L.phase = PH_IDLE;
  Tally T = tally_new();
  bool exhausted = false;
  for (;;) {
    unsigned idle = __ballot_sync(0xffffffffu, L.phase == PH_IDLE);
    int nidle = __popc(idle);
    if (!exhausted && (nidle >= refill || nidle == 32) && nidle > 0) {
      unsigned long long b = 0;
      if (lane == 0) b = atomicAdd(queue, (unsigned long long)nidle);
      b = __shfl_sync(0xffffffffu, b, 0);
      if (b + (unsigned long long)nidle >= total) exhausted = true;
      if (L.phase == PH_IDLE) {
        unsigned long long w = b + (unsigned long long)__popc(idle & lt_mask);
        if (w < total) lane_start<PASS_BOTH>(L, reqs, base, n_req, w, true);
      }
    }
    unsigned active = __ballot_sync(0xffffffffu, L.phase != PH_IDLE);
    if (active == 0) {
      if (exhausted) break;
      continue;
    }
    if (L.phase != PH_IDLE) lane_advance<FULL, PASS_BOTH>(L, reqs, K, T);
  }
  tally_flush(T, reqs);
}

}  // namespace

}  // namespace jsh

using namespace jsh;

#if JSH_FARADAY_THICK_BUILD
#define JSH_STATIC_KERNEL jsh_static_kernel_ft
#define JSH_SINGLE_KERNEL jsh_single_kernel_ft
#else
#define JSH_STATIC_KERNEL jsh_static_kernel
#define JSH_SINGLE_KERNEL jsh_single_kernel
#endif
StaticKernel JSH_STATIC_KERNEL(bool full) {
  return full ? transfer_static_mixed_kernel<true> : transfer_static_mixed_kernel<false>;
}
SingleKernel JSH_SINGLE_KERNEL(bool full, bool compact) {
  if (compact) return full ? transfer_persistent_mixed_kernel<true, true> : transfer_persistent_mixed_kernel<false, true>;
  return full ? transfer_persistent_mixed_kernel<true, false> : transfer_persistent_mixed_kernel<false, false>;
}
