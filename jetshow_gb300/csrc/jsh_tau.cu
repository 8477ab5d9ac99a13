// jsh_tau.cu -- the split form's first half: the heaviest-first ranking of the
// hit rays, the tau kernels, and the ranking of the items they hand on.  The
// Faraday-thick mode of the IQUV pass does not reach this code, so both
// launch sequences (jsh_persistent.cu and its second build) share it.
#include <algorithm>

#include "jsh_mixed.cuh"

#include "jsh_split.h"

namespace jsh {

namespace {

// ------------------------------------------------------------- ranking
// Heaviest-first order of the hit rays for the persistent schedule.  A ray's
// cost grows with its optical depth (up to the optically thick start of the
// IQUV pass): rays through the core take thousands of steps, rays far out a
// few hundred.  So each ray's optical depth at the request's first
// frequency is estimated (4-point Gauss-Legendre over each segment, the FP32
// coefficients), bucketed by factors of 2 and counting-sorted in descending
// order; the queue then hands out the heaviest rays first and they run while
// the bulk fills the GPU, instead of starting late and setting the render's
// makespan.
template <bool ANY>
__global__ void __launch_bounds__(256) rank_cost_kernel(const JshRequest* __restrict__ reqs) {
  __shared__ uint32_t hist[JSH_RANK_BUCKETS];
  const JshRequest& R = reqs[blockIdx.y];
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h < *R.n_hit) {
    const JshHit& H = R.hits[h];
    const JshFreqConst F = R.mix.fc[0];
    const float xk[4] = {0.0694318442f, 0.330009478f, 0.669990522f, 0.930568156f};
    const float wk[4] = {0.173927423f, 0.326072577f, 0.326072577f, 0.173927423f};
    float tau = 0.f;
    for (int s = 0; s < H.nseg && s < 2; ++s) {
      const JshSeg32& S = segment_of<ANY>(R, h, s);
      const F3 a = f3(S.in[0], S.in[2], S.in[4]), b = f3(S.out[0], S.out[2], S.out[4]);
      const F3 d = b - a;
      float acc = 0.f;
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        Coef32 c;
        coef32_rt(R, R.mix, F, a + d * xk[k], COEF_KI, c);
        acc = fmaf(wk[k], c.kI, acc);
      }
      tau = fmaf(acc, sqrtf(fdot(d, d)), tau);
    }
    int key = 0;
    if (tau > 0.f && tau < INFINITY) key = min(max((int)floorf(__log2f(tau)) + 40, 1), JSH_RANK_BUCKETS - 1);
    R.key[h] = (uint8_t)key;
    atomicAdd(&hist[key], 1u);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x)
    if (hist[b]) atomicAdd(&R.buckets[b], hist[b]);
}

// Start of each bucket in descending bucket order (one thread per request),
// and the size of the deep prefix: the rays of buckets >= deep_key (every
// ray for deep_key <= 0).
__global__ void rank_prefix_kernel(const JshRequest* __restrict__ reqs, int deep_key) {
  const JshRequest& R = reqs[blockIdx.x];
  if (threadIdx.x != 0) return;
  uint32_t run = 0, deep = 0;
  for (int b = JSH_RANK_BUCKETS - 1; b >= 0; --b) {
    R.buckets[JSH_RANK_BUCKETS + b] = run;
    run += R.buckets[b];
    if (b == deep_key) deep = run;
  }
  R.buckets[JSH_RANK_DEEP] = deep_key > 0 ? deep : run;
}

// order[position] = hit index; the lanes of a warp with the same bucket take
// consecutive positions with one atomic.
__global__ void __launch_bounds__(256) rank_scatter_kernel(const JshRequest* __restrict__ reqs) {
  const JshRequest& R = reqs[blockIdx.y];
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= *R.n_hit) return;
  const int key = R.key[h];
  const unsigned peers = __match_any_sync(__activemask(), key);
  const int leader = __ffs(peers) - 1;
  const unsigned lane = threadIdx.x & 31u;
  uint32_t base = 0;
  if ((int)lane == leader) base = atomicAdd(&R.buckets[JSH_RANK_BUCKETS + key], (uint32_t)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  R.order[base + __popc(peers & ((1u << lane) - 1u))] = h;
}

// ------------------------------------------------------------ split form
// The persistent schedule's default form runs the passes in two kernels:
// every item's tau pass first (one stage component, k_I only: a short
// right-hand side, few registers, many resident warps, and no warp whose
// lanes mix tau and IQUV code), then the I/IQUV pass of the items that need
// one, ranked by the optical depth it integrates through.

// Work items of part `part` of the ranked rays over the batch (exclusive
// prefix in shared memory): part 0 the deep prefix (every ray when the
// passes are not overlapped), part 1 the rays after it.
__device__ __forceinline__ void tau_prefix(const JshRequest* __restrict__ reqs, int n_req, int part,
                                           unsigned long long* base) {
  if (threadIdx.x == 0) {
    unsigned long long acc = 0;
    for (int r = 0; r < n_req; ++r) {
      base[r] = acc;
      const uint32_t deep = reqs[r].buckets[JSH_RANK_DEEP];
      const uint32_t rays = part ? *reqs[r].n_hit - deep : deep;
      acc += (unsigned long long)rays * (unsigned long long)reqs[r].n_nu;
    }
    base[n_req] = acc;
  }
  __syncthreads();
}

// Tau kernels: persistent CTAs, lanes (or groups of lanes) refilled from the
// ranked queue (the same order as the single-kernel form), each item's tau
// pass to its end, over the rays of part `part`.
//
// The build for batches of the fused benchmark family alone (80 registers, 24
// resident warps per SM).  Up to kTauGroupsFused items per group of the grid
// (88 000 on 152 SMs) they run on groups: a panel is three evaluations' time
// instead of fifteen, which counts while rays are few (2 022 items 129 -> 50
// us, 32 350 items 160 -> 80 us, 79 782 items 174 -> 165 us); above, a lane
// each does less work per panel (129 394 items 201 us against 227 us on
// groups, 705 176 items 555 against 1 155 us).
//
// ONE: a launch on a single request, whose constants (`mix`) are the kernel's
// parameters and so operands of its instructions; otherwise each lane loads
// them from its request's record, again for every node at 80 registers (a
// batch cannot do else).  512x1024 x 4: 522 -> 430 us.  The IQUV kernel, whose
// step is more code than the instruction caches hold, loses by it (1.39 -> 1.56
// ms): constants and instructions share a cache.
constexpr int kTauGroupsFused = 4;
template <bool ONE>
__global__ void __launch_bounds__(256, 3)
    transfer_tau_kernel(const JshRequest* __restrict__ reqs, int n_req, unsigned long long* queue, int refill,
                        int part, const __grid_constant__ JshMixed mix) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  tau_prefix(reqs, n_req, part, base);
  Lane L;
  L.phase = PH_IDLE;
  Tally T = tally_new();
  const unsigned long long total = base[n_req];
  auto start = [&](unsigned long long w) {
    lane_start<PASS_TAU>(L, reqs, base, n_req, w, true, part, ONE ? &mix : nullptr);
  };
  if (on_groups(total, kTauGroupsFused)) {
    const LaneGroup grp = lane_group();
    run_queue(L, queue, total, refill, grp, true, false, 0, start,
              [&] { tau_step<PASS_TAU, false, kGroupLanes>(L, reqs, ONE ? mix : reqs[L.r].mix, nullptr, part, T, grp); });
  } else {
    const LaneGroup one = single_lane();
    run_queue(L, queue, total, refill, one, false, false, 0, start,
              [&] { tau_step<PASS_TAU, false, 1>(L, reqs, ONE ? mix : reqs[L.r].mix, nullptr, part, T, one); });
  }
  tally_flush(T, reqs);
}

// The build for every field law, with a lane per item (128 registers, 16
// resident warps per SM) or a group per item (the same: at 161 registers and 12
// warps 29 092 items of a radial field took 211 us, now 174, a simulation grid at
// 256^2 19.6 ms, now 19.1; at 102 registers and 20 warps 195 us and 21.4 ms).
template <bool GROUPS>
__global__ void __launch_bounds__(128, 4)
    transfer_tau_general_kernel(const JshRequest* __restrict__ reqs, int n_req, unsigned long long* queue, int refill,
                                int part, const __grid_constant__ JshMixed /* the fused build's alone */) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  extern __shared__ float ksh[];
  tau_prefix(reqs, n_req, part, base);
  Lane L;
  L.phase = PH_IDLE;
  Tally T = tally_new();
  const LaneGroup grp = GROUPS ? lane_group() : single_lane();
  float* K = ksh + (GROUPS ? group_slot(grp) : (int)threadIdx.x) * kTauWords;
  run_queue(
      L, queue, base[n_req], refill, grp, GROUPS, false, 0,
      [&](unsigned long long w) { lane_start<PASS_TAU>(L, reqs, base, n_req, w, true, part); },
      [&] { tau_step<PASS_TAU, true, 0>(L, reqs, reqs[L.r].mix, K, part, T, grp); });
  tally_flush(T, reqs);
}

// Cost histogram of part `part`'s emitted items of request blockIdx.y
// (grid-stride), and the items' FP64 work, a full warp of them at a time: the
// tau plane where the depth is still a pair, the first-step divisor.
__global__ void __launch_bounds__(256) iquv_hist_kernel(const JshRequest* __restrict__ reqs, int part) {
  __shared__ uint32_t hist[JSH_RANK_BUCKETS];
  const JshRequest& R = reqs[blockIdx.y];
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  const uint32_t n = R.iq_count[part], o = iq_first(R, part);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    JshIquvItem& it = R.iq_items[o + i];
    atomicAdd(&hist[it.key], 1u);
    double tau = it.tau_bg;
    if (it.flags & 32) {
      tau = df_val(DF{it.tau_pair[0], it.tau_pair[1]});
      if (R.tau) R.tau[(uint64_t)it.f * R.npix + (uint64_t)R.hits[it.h].pix] = tau;
    }
    it.first_div = first_step_divisor(tau, R.P.n);
  }
  __syncthreads();
  uint32_t* bk = R.iq_buckets + 2 * JSH_RANK_BUCKETS * part;
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x)
    if (hist[b]) atomicAdd(&bk[b], hist[b]);
}

// Start of each cost bucket in descending order (one thread per request).
__global__ void iquv_prefix_kernel(const JshRequest* __restrict__ reqs, int part) {
  const JshRequest& R = reqs[blockIdx.x];
  if (threadIdx.x != 0) return;
  uint32_t* bk = R.iq_buckets + 2 * JSH_RANK_BUCKETS * part;
  uint32_t run = 0;
  for (int b = JSH_RANK_BUCKETS - 1; b >= 0; --b) {
    bk[JSH_RANK_BUCKETS + b] = run;
    run += bk[b];
  }
}

// iq_order[first + position] = emitted item (absolute slot).  Each CTA takes a
// stretch of the items, counts its keys in shared memory, reserves its part of
// every bucket with one global atomic and hands the positions out in shared
// memory: an atomic per key and warp on 64 addresses took 40 us of a 512x1024
// render of 4 frequencies.
__global__ void __launch_bounds__(256) iquv_scatter_kernel(const JshRequest* __restrict__ reqs, int part) {
  __shared__ uint32_t count[JSH_RANK_BUCKETS], next[JSH_RANK_BUCKETS];
  const JshRequest& R = reqs[blockIdx.y];
  const uint32_t n = R.iq_count[part], o = iq_first(R, part);
  const uint32_t each = (n + gridDim.x - 1) / gridDim.x;
  const uint32_t i0 = min(n, blockIdx.x * each), i1 = min(n, i0 + each);
  if (i0 == i1) return;
  uint32_t* bk = R.iq_buckets + 2 * JSH_RANK_BUCKETS * part;
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x) count[b] = 0;
  __syncthreads();
  for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) atomicAdd(&count[R.iq_items[o + i].key], 1u);
  __syncthreads();
  for (int b = threadIdx.x; b < JSH_RANK_BUCKETS; b += blockDim.x)
    next[b] = count[b] ? atomicAdd(&bk[JSH_RANK_BUCKETS + b], count[b]) : 0u;
  __syncthreads();
  for (uint32_t i = i0 + threadIdx.x; i < i1; i += blockDim.x)
    R.iq_order[o + atomicAdd(&next[R.iq_items[o + i].key], 1u)] = o + i;
}

}  // namespace

}  // namespace jsh

using namespace jsh;

TauLaunch jsh_tau_kernel(bool fused, bool groups, bool one) {
  if (fused) return TauLaunch{one ? transfer_tau_kernel<true> : transfer_tau_kernel<false>, 256, 0};
  return TauLaunch{groups ? transfer_tau_general_kernel<true> : transfer_tau_general_kernel<false>, 128,
                   sizeof(float) * kTauWords * (groups ? 128 / 32 * kWarpGroups : 128)};
}

void jsh_launch_rank(const JshRequest* d_reqs, int n_req, uint64_t max_hits, int deep_key, bool seg32,
                     cudaStream_t stream) {
  const dim3 g((unsigned)((max_hits + 255) / 256), (unsigned)n_req);
  if (seg32) rank_cost_kernel<false><<<g, 256, 0, stream>>>(d_reqs);
  else rank_cost_kernel<true><<<g, 256, 0, stream>>>(d_reqs);
  rank_prefix_kernel<<<n_req, 32, 0, stream>>>(d_reqs, deep_key);
  rank_scatter_kernel<<<g, 256, 0, stream>>>(d_reqs);
}

void jsh_launch_iquv_rank(const JshRequest* d_reqs, int n_req, uint64_t max_items, int num_sms, int part,
                          cudaStream_t stream) {
  // enough CTAs in flight to hide the gathers' latency, none without items
  const uint64_t each = (max_items / (uint64_t)n_req + 255) / 256;
  const dim3 g((unsigned)std::min<uint64_t>(std::max<uint64_t>(each, 1), 4 * (uint64_t)num_sms), (unsigned)n_req);
  iquv_hist_kernel<<<g, 256, 0, stream>>>(d_reqs, part);
  iquv_prefix_kernel<<<n_req, 32, 0, stream>>>(d_reqs, part);
  iquv_scatter_kernel<<<g, 256, 0, stream>>>(d_reqs, part);
}
