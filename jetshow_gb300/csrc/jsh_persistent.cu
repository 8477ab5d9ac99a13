// jsh_persistent.cu -- the mixed path's launch sequence and the split form's
// second half, the IQUV kernels (the lane machine is jsh_mixed.cuh, the
// ranking and tau kernels are jsh_tau.cu, the other forms jsh_forms.cu).
//
// This file is compiled twice: as is, and by jsh_persistent_ft.cu with
// JSH_FARADAY_THICK_BUILD 1 for requests that ask for the Faraday-thick mode.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "jsh_mixed.cuh"

#include "jsh_context.h"
#include "jsh_split.h"

#if JSH_FARADAY_THICK_BUILD
#define JSH_LAUNCH_TRANSFER_MIXED jsh_launch_transfer_mixed_ft
#define JSH_MIXED_OCCUPANCY jsh_mixed_occupancy_ft
#define JSH_STATIC_KERNEL jsh_static_kernel_ft
#define JSH_SINGLE_KERNEL jsh_single_kernel_ft
#else
#define JSH_LAUNCH_TRANSFER_MIXED jsh_launch_transfer_mixed
#define JSH_MIXED_OCCUPANCY jsh_mixed_occupancy
#define JSH_STATIC_KERNEL jsh_static_kernel
#define JSH_SINGLE_KERNEL jsh_single_kernel
#endif

namespace jsh {

namespace {

// Exclusive prefix of part `part`'s emitted items over the batch, in shared
// memory.
__device__ __forceinline__ void iquv_prefix(const JshRequest* __restrict__ reqs, int n_req, int part,
                                            unsigned long long* base) {
  if (threadIdx.x == 0) {
    unsigned long long acc = 0;
    for (int r = 0; r < n_req; ++r) {
      base[r] = acc;
      acc += (unsigned long long)reqs[r].iq_count[part];
    }
    base[n_req] = acc;
  }
  __syncthreads();
}

// IQUV kernels: persistent CTAs over the ranked emitted items.
//
// The build for the fused benchmark family alone (128 registers, 16 resident
// warps per SM; with the Faraday-thick mode 145 and 12; there is no
// register-capped build of it: capped at the same 16 warps it held 124 and was
// 1.2 % slower).  With many items they run on a
// lane each, dealt so that the longest are in different warps, and once the
// queue is empty a warp's last six are handed to its groups of lanes, which
// take a step in under half the time: the longest items decide when the launch
// ends (the longest of 517 856 Faraday-thick items has 21 000 evaluations: 11.8
// -> 9.1 ms; 129 468 of them 11.2 -> 6.6 ms; 129 394 items of a conical jet 430
// -> 345 us, 517 550 1.10 -> 0.91 ms; 705 176 of a longer-tailed image 1.42 ms
// before and after, bound by the step's instructions).  Without the dealing the
// longest are one warp's and the 517 856 items take 12.8 ms; handing over the
// last three only, 11.8.
//
// Up to kIquvGroups* items per group of the grid they run on groups from the
// start: 8 092 items 86 us on lanes, 74 on groups.  Above, lanes have the
// better throughput: 32 350 items 221 against 236 us, 79 782 items 639 against
// 713; in the Faraday-thick build 32 368 items 5.5 against 5.2 ms, 50 572 items
// 6.15 against 6.23; Stokes I alone 2 022 items 43 us on either.
static_assert(kWarpGroups * kGroupWords <= 32 * kLaneWords, "a warp's groups fit its lanes' storage");
constexpr int kIquvGroupsFull = kFtm ? 4 : 2, kIquvGroupsI = 1;
template <bool FULL>
__global__ void __launch_bounds__(256, 1)
    transfer_iquv_kernel(const JshRequest* __restrict__ reqs, int n_req, unsigned long long* queue, int refill,
                         int part) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  extern __shared__ __align__(16) float ksh[];
  iquv_prefix(reqs, n_req, part, base);
  Lane L;
  L.phase = PH_IDLE;
  Tally T = tally_new();
  const unsigned long long total = base[n_req];
  auto start = [&](unsigned long long w) { lane_start_iquv<false>(L, reqs, base, n_req, w, part); };
  const LaneGroup grp = lane_group(), one = single_lane();
  // a warp's lanes and groups share its part of the storage (full Stokes)
  float* W = ksh + threadIdx.x / 32 * 32 * kLaneWords;
  float* Q = FULL ? W + min(grp.base / kGroupLanes, kWarpGroups - 1) * kGroupWords : ksh + group_slot(grp) * kGroupWords;
  auto group_step = [&] { lane_step<FULL, PASS_IQUV, false, kGroupLanes>(L, reqs, reqs[L.r].mix, Q, T, grp); };
  const bool lanes = !on_groups(total, FULL ? kIquvGroupsFull : kIquvGroupsI);
  if (lanes) {
    run_queue(L, queue, total, refill, one, true, false, kWarpGroups, start,
              [&] { lane_step<FULL, PASS_IQUV, false, 1>(L, reqs, reqs[L.r].mix, W + (threadIdx.x & 31u) * kLaneWords, T, one); });
    spread_items(L, grp);
  }
  run_queue(L, queue, total, refill, grp, !lanes, lanes, 0, start, group_step);
  tally_flush(T, reqs);
}

// The build for every field law, with a lane or a group of lanes per item.
template <bool FULL, bool COMPACT, bool GROUPS>
__global__ void __launch_bounds__(COMPACT || GROUPS ? 128 : 256, COMPACT || GROUPS ? 3 : 1)
    transfer_iquv_general_kernel(const JshRequest* __restrict__ reqs, int n_req, unsigned long long* queue, int refill,
                                 int part) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  extern __shared__ __align__(16) float ksh[];
  iquv_prefix(reqs, n_req, part, base);
  Lane L;
  L.phase = PH_IDLE;
  Tally T = tally_new();
  const LaneGroup grp = GROUPS ? lane_group() : single_lane();
  float* Q = ksh + (GROUPS ? group_slot(grp) : (int)threadIdx.x) * StageWidth<FULL>::kWords;
  run_queue(
      L, queue, base[n_req], refill, grp, GROUPS, false, 0,
      [&](unsigned long long w) { lane_start_iquv<true>(L, reqs, base, n_req, w, part); },
      [&] { lane_step<FULL, PASS_IQUV, true, 0>(L, reqs, reqs[L.r].mix, Q, T, grp); });
  tally_flush(T, reqs);
}

// Lets `kernel` take `smem` bytes of stage storage.  A launch gets 48 KB unasked,
// static storage included, and a full-Stokes lane of the every-law and
// single-kernel builds keeps 196 bytes: 256 threads take 50 176.  Where it has
// to be asked for, always the same bytes are, the largest CTA's: launches of
// several threads do not lower each other's limit.
template <typename K>
cudaError_t allow_storage(K kernel, size_t smem) {
  constexpr size_t kUnasked = (48u << 10) - 1024;
  if (smem <= kUnasked) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage_smem<true>(256));
}

template <typename K>
int occupancy(K kernel, int block, size_t smem) {
  int n = 0;
  if (allow_storage(kernel, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, block, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace

}  // namespace jsh

using namespace jsh;

namespace jsh {
namespace {

// Registers a warp of `kernel` holds (allocated in units of 256), looked up
// once per kernel.
template <typename K>
int warp_regs(K kernel) {
  static std::mutex mu;
  static std::unordered_map<const void*, int> known;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find((const void*)kernel);
  if (it != known.end()) return it->second;
  cudaFuncAttributes a;
  const int w = cudaFuncGetAttributes(&a, kernel) == cudaSuccess ? (a.numRegs * 32 + 255) / 256 * 256 : 255 * 32;
  known[(const void*)kernel] = w;
  return w;
}

// Launch with a per-launch scheduling priority (the overlapped deep chain).
template <typename... KArgs, typename... Args>
cudaError_t launch_prio(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                        int prio, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributePriority;
  at[0].val.priority = prio;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Work items up to which the kernels for every law put each on a group of
// lanes, per SM (the host knows the pixels, not the hits: an upper bound; 57 %
// of these images hit).  Groups against lanes [ms], tau + IQUV kernel of square
// images at one frequency, 152 SMs:
//   pixels  items/SM  grid of 200 000 points  sheath flow   radial field
//   256^2     431     25.2 + 16.8, 36.1 + 16.3  0.52 + 0.53, 1.17 + 0.93  0.27 + 0.20, 0.31 + 0.23
//   300^2     592     32.5 + 22.5, 36.5 + 23.3  0.66 + 0.67, 1.20 + 0.92  0.34 + 0.27, 0.30 + 0.30
//   360^2     853     44.5 + 31.6, 37.4 + 27.6  0.83 + 0.87, 1.19 + 1.20  0.48 + 0.39, 0.29 + 0.38
//   512^2    1725     85.3 + 62.2, 63.7 + 49.9  1.39 + 1.53, 1.48 + 1.39  0.94 + 0.77, 0.53 + 0.59
// Both kernels change sides between 300^2 and 360^2 on grids, the radial field
// at 256^2 to 360^2, the sheath at 512^2; Stokes I alone the same or earlier (radial field 0.17
// against 0.12 ms at 256^2, sheath 0.55 against 0.95 at 300^2).  The line lies
// between the two sizes at which the grids change.
constexpr uint64_t kGroupItemsPerSm = 720;

// IQUV kernel instantiation of a launch.
IquvKernel iquv_kernel(bool full, bool compact, bool fused, bool groups) {
  if (fused) return full ? transfer_iquv_kernel<true> : transfer_iquv_kernel<false>;
  if (groups) return full ? transfer_iquv_general_kernel<true, false, true> : transfer_iquv_general_kernel<false, false, true>;
  if (compact)
    return full ? transfer_iquv_general_kernel<true, true, false> : transfer_iquv_general_kernel<false, true, false>;
  return full ? transfer_iquv_general_kernel<true, false, false> : transfer_iquv_general_kernel<false, false, false>;
}

// The IQUV kernel of a split launch on at most `items` work items.
struct IquvLaunch {
  IquvKernel kernel;
  bool groups, full, fused;
  // most threads a CTA of it can have
  int max_block(bool compact) const { return compact || groups ? 128 : 256; }
  // the fused build: a lane keeps its five points (full Stokes) or nothing there
  size_t smem(int block) const { return full ? stage_smem<true>(block, !fused) : stage_smem<false>(block, !fused); }
};
IquvLaunch iquv_launch(bool full, const JshLaunchShape& shape, uint64_t items, int num_sms) {
  const bool fused = shape.fused != 0, groups = !fused && items <= kGroupItemsPerSm * (uint64_t)num_sms;
  return IquvLaunch{iquv_kernel(full, shape.compact != 0, fused, groups), groups, full, fused};
}

// CTAs of the deep chain's IQUV kernel per SM (64 threads each) when the
// passes overlap: room for the deep prefix's longest items from the start,
// the rest of the SM for the other rays' tau kernel.
constexpr int kDeepIquvBlock = 64;
constexpr int kDeepIquvPerSm = 2;

}  // namespace
}  // namespace jsh

cudaError_t JSH_LAUNCH_TRANSFER_MIXED(const JshRequest* d_reqs, int n_req, int schedule, bool full,
                                      uint64_t max_items, uint64_t max_hits, const JshLaunchShape& shape,
                                      unsigned int* queue, int num_sms, cudaStream_t stream) {
  if (schedule == JSH_SCHED_STATIC) {
    const int bs = 128;
    unsigned blocks = (unsigned)((max_items + bs - 1) / bs);
    JSH_STATIC_KERNEL(full)<<<blocks, bs, full ? stage_smem<true>(bs) : stage_smem<false>(bs), stream>>>(d_reqs, n_req);
    return cudaGetLastError();
  }
  const bool split = !shape.single;
  const bool overlap = split && shape.overlap_key > 0 && shape.side != nullptr && shape.fork != nullptr;
  if (max_hits > 0) jsh_launch_rank(d_reqs, n_req, max_hits, overlap ? shape.overlap_key : 0, split, stream);
  // queue counters: [0] tau (deep prefix or all) / single-kernel form, [1]
  // its IQUV kernel, [2] and [3] the other rays' tau and IQUV kernels
  unsigned long long* q = (unsigned long long*)queue;
  const uint64_t need = (max_items + 31) / 32 * 32;
  const int rf = shape.refill_threshold;
  int bs = shape.block_size;
  if (bs > (shape.compact ? 128 : 256)) bs = shape.compact ? 128 : 256;
  if (!split) {
    const SingleKernel kernel = JSH_SINGLE_KERNEL(full, shape.compact != 0);
    const size_t smem = full ? stage_smem<true>(bs) : stage_smem<false>(bs);
    const cudaError_t e = allow_storage(kernel, smem);
    if (e != cudaSuccess) return e;
    const int per_sm = shape.ctas_per_sm > 0 ? shape.ctas_per_sm : occupancy(kernel, bs, smem);
    unsigned blocks = (unsigned)(num_sms * std::max(per_sm, 1));
    if ((uint64_t)blocks * bs > need) blocks = (unsigned)((need + bs - 1) / bs);
    if (blocks == 0) blocks = 1;
    if (shape.marks) cudaEventRecord(shape.marks[2], stream);
    kernel<<<blocks, bs, smem, stream>>>(d_reqs, n_req, q, rf);
    if (shape.marks) cudaEventRecord(shape.marks[3], stream);
    return cudaGetLastError();
  }
  // tau kernel: 256 threads, every CTA it can keep resident (the fused build
  // runs panels only, which keep their sums in registers; the general build
  // keeps Dormand-Prince stages in shared memory)
  const IquvLaunch iquv = iquv_launch(full, shape, need, num_sms);
  const bool one = shape.mix != nullptr && n_req == 1;
  const JshMixed mix = one ? *shape.mix : JshMixed{};
  const TauLaunch tau = jsh_tau_kernel(shape.fused != 0, iquv.groups, one);
  const TauKernel tau_k = tau.kernel;
  const int bt = tau.block;
  const size_t smem_t = tau.smem;
  int per_sm_t = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_t, tau_k, bt, smem_t);
  if (per_sm_t < 1) per_sm_t = 1;
  unsigned bl_t = (unsigned)(num_sms * per_sm_t);
  // a CTA holds fewer items on groups of lanes than on single ones: enough
  // CTAs for the former
  auto enough = [&](unsigned grid, int block) {
    const unsigned per_cta = (unsigned)(block / 32 * kWarpGroups);
    return (unsigned)std::min<uint64_t>(grid, (need + per_cta - 1) / per_cta);
  };
  bl_t = enough(bl_t, bt);
  const IquvKernel iquv_k = iquv.kernel;
  bs = std::min(bs, iquv.max_block(shape.compact != 0));
  const size_t smem_q = iquv.smem(bs);
  cudaError_t e = allow_storage(iquv_k, smem_q);
  if (e != cudaSuccess) return e;
  int per_sm_q = shape.ctas_per_sm;
  if (per_sm_q <= 0) per_sm_q = occupancy(iquv_k, bs, smem_q);
  const unsigned blocks_q = enough((unsigned)(num_sms * std::max(per_sm_q, 1)), bs);
  if (!overlap) {
    if (shape.marks) cudaEventRecord(shape.marks[0], stream);
    tau_k<<<bl_t, bt, smem_t, stream>>>(d_reqs, n_req, q, rf, 0, mix);
    if (shape.marks) cudaEventRecord(shape.marks[1], stream);
    jsh_launch_iquv_rank(d_reqs, n_req, max_items, num_sms, 0, stream);
    if (shape.marks) cudaEventRecord(shape.marks[2], stream);
    iquv_k<<<blocks_q, bs, smem_q, stream>>>(d_reqs, n_req, q + 1, rf, 0);
    if (shape.marks) cudaEventRecord(shape.marks[3], stream);
    return cudaGetLastError();
  }
  // Overlapped passes.  Deep chain on `stream`: the deep prefix's tau pass
  // on the whole GPU, its IQUV ranking, then its IQUV kernel at high
  // priority on kDeepIquvPerSm small CTAs per SM.  The other rays' chain on
  // `side` starts when the deep IQUV kernel becomes ready (the fork event
  // follows its ranking), with as many tau CTAs per SM as fit beside the
  // deep IQUV CTAs, so that the deep items start at once and the two chains
  // share every SM.  Neither chain waits on the other inside a kernel.
  static const int prio_hi = [] {
    int least = 0, greatest = 0;
    return cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess ? greatest : 0;
  }();
  const int wr_iquv = warp_regs(iquv_k), wr_tau = warp_regs(tau_k);
  const int deep_warps = kDeepIquvPerSm * kDeepIquvBlock / 32;
  int per_sm_t2 = (65536 - deep_warps * wr_iquv) / ((bt / 32) * wr_tau);
  per_sm_t2 = std::min(std::max(per_sm_t2, 1), per_sm_t);
  if (shape.marks) cudaEventRecord(shape.marks[0], stream);
  e = launch_prio(tau_k, bl_t, bt, smem_t, stream, prio_hi, d_reqs, n_req, q, rf, 0, mix);
  if (e != cudaSuccess) return e;
  jsh_launch_iquv_rank(d_reqs, n_req, max_items, num_sms, 0, stream);
  e = cudaEventRecord(shape.fork[0], stream);
  if (e != cudaSuccess) return e;
  e = launch_prio(iquv_k, (unsigned)(num_sms * kDeepIquvPerSm), kDeepIquvBlock,
                  iquv.smem(kDeepIquvBlock), stream, prio_hi,
                  d_reqs, n_req, q + 1, rf, 0);
  if (e != cudaSuccess) return e;
  e = cudaStreamWaitEvent(shape.side, shape.fork[0], 0);
  if (e != cudaSuccess) return e;
  unsigned bl_t2 = (unsigned)(num_sms * per_sm_t2);
  bl_t2 = enough(bl_t2, bt);
  tau_k<<<bl_t2, bt, smem_t, shape.side>>>(d_reqs, n_req, q + 2, rf, 1, mix);
  if (shape.marks) cudaEventRecord(shape.marks[1], shape.side);
  jsh_launch_iquv_rank(d_reqs, n_req, max_items, num_sms, 1, shape.side);
  if (shape.marks) cudaEventRecord(shape.marks[2], shape.side);
  iquv_k<<<blocks_q, bs, smem_q, shape.side>>>(d_reqs, n_req, q + 3, rf, 1);
  e = cudaEventRecord(shape.fork[1], shape.side);
  if (e != cudaSuccess) return e;
  e = cudaStreamWaitEvent(stream, shape.fork[1], 0);
  if (e != cudaSuccess) return e;
  if (shape.marks) cudaEventRecord(shape.marks[3], stream);
  return cudaGetLastError();
}

// Resident CTAs per SM of `block` threads of the kernel that a request of at most
// `items` work items runs with `shape`: the IQUV kernel of the split form, or the
// single-kernel form; 0 if it cannot run them.
int JSH_MIXED_OCCUPANCY(bool full, int block, const JshLaunchShape& shape, uint64_t items, int num_sms) {
  if (shape.single) {
    if (block > (shape.compact ? 128 : 256)) return 0;
    return occupancy(JSH_SINGLE_KERNEL(full, shape.compact != 0), block,
                     full ? stage_smem<true>(block) : stage_smem<false>(block));
  }
  const IquvLaunch iquv = iquv_launch(full, shape, (items + 31) / 32 * 32, num_sms);  // as the launch rounds them
  return block > iquv.max_block(shape.compact != 0) ? 0 : occupancy(iquv.kernel, block, iquv.smem(block));
}

#if !JSH_FARADAY_THICK_BUILD  // the host functions below are built once
int jsh_queue64_occupancy(int block_size);
int jsh_mixed_occupancy_ft(bool full, int block, const JshLaunchShape& shape, uint64_t items, int num_sms);

int jsh_persistent_occupancy(int precision, bool full, int block_size, const JshLaunchShape& shape, uint64_t items,
                             int num_sms) {
  if (precision != JSH_PREC_MIXED) return jsh_queue64_occupancy(block_size);
  return full && shape.faraday_thick ? jsh_mixed_occupancy_ft(full, block_size, shape, items, num_sms)
                                     : jsh_mixed_occupancy(full, block_size, shape, items, num_sms);
}

// ------------------------------------------------------------------ host
// Per-request and per-frequency constants of the FP32 coefficient algebra,
// evaluated in FP64 from the compiled model.
int jsh_prepare_mixed(JshRequest* req, const double* nu_host, JshFreqConst* fc) {
  const JshModel& m = req->model;
  JshMixed& X = req->mix;
  const JshFreqConst* keep = X.fc;
  memset(&X, 0, sizeof(X));
  X.fc = keep;
  const double s = m.s;
  const double nx = -req->plane.dx, ny = -req->plane.dy, nz = -req->plane.dz;
  X.nl[0] = (float)nx;
  X.nl[1] = (float)ny;
  X.nl[2] = (float)nz;
  X.pk = (float)((s + 2.) / 2.);
  X.dt_max_pc = req->P.dt_max / JSH_PC;
  X.dt_max_f = (float)X.dt_max_pc;
  X.tau_min_f = nextafterf((float)(std::max(req->P.tau_min, 0.0) * (1.0 + 1e-6)), INFINITY);
  {
    const double d[3] = {req->plane.dx, req->plane.dy, req->plane.dz};
    for (int k = 0; k < 3; ++k) {
      X.dhi[k] = (float)d[k];
      X.dlo[k] = (float)(d[k] - (double)X.dhi[k]);
    }
    X.tau_max_hi = (float)req->P.tau_max;
    X.tau_max_lo = (float)(req->P.tau_max - (double)X.tau_max_hi);
  }
  X.tau_atol = (float)req->P.tau_atol;
  X.tau_rtol = (float)req->P.tau_rtol;
  X.rtol = (float)req->P.rtol;
  X.kq = (float)m.kq_ratio;
  X.eq = (float)m.eq_ratio;
  X.sim_shared = (m.v_kind == JSH_V_SIMULATION && m.n_kind == JSH_N_SIMULATION && m.b_kind == JSH_B_SIMULATION &&
                  m.grid_v == m.grid_b && m.grid_n == m.grid_b)
                     ? 1
                     : 0;
  for (int i = 0; i < 8; ++i) {
    X.vq[i] = (float)m.vp[i];
    X.vq_pc[i] = (float)(m.vp[i] / JSH_PC);
    X.nq[i] = (float)m.np[i];
    X.nq_pc[i] = (float)(m.np[i] / JSH_PC);
    X.bq[i] = (float)m.bp[i];
    X.bq_pc[i] = (float)(m.bp[i] / JSH_PC);
  }
  X.v_dq01 = (float)(m.vp[0] - m.vp[1]);
  X.v_g0m1 = (float)(m.vp[0] - 1.0);
  X.v_cone_oz = (float)m.v_cone_oz;
  X.v_cone_oz_pc = (float)(m.v_cone_oz / JSH_PC);
  X.v_theta = (float)m.v_theta;
  X.v_omc = (float)(2.0 * sin(0.5 * m.vp[2]) * sin(0.5 * m.vp[2]));
  X.sin_pitch = (float)m.sin_pitch;
  X.cos_pitch = (float)m.cos_pitch;
  X.tan_pitch = (float)m.tan_pitch;
  X.b_bessel0 = (float)(m.bp[0] * m.bessel0);
  X.b_bessel1 = (float)(m.bp[0] * m.bessel1);
  // optically thick start of the IQUV pass: the Stokes vector decays at
  // least at rate k_I (1 - |(k_Q, k_U, k_V)| / k_I) along the ray (the
  // symmetric part of the transfer matrix; Faraday terms only rotate), so
  // what enters at optical depth tau_thick is attenuated by exp(-16)
  {
    double p = req->P.full ? std::min(0.95, m.kq_ratio + 0.05) : 0.0;
    double thick = 16.0 / (1.0 - p);
    X.tau_thick = (req->P.flags & JSH_FLAG_IQUV_FROM_TAU_MAX) || !(thick < req->P.tau_max) ? INFINITY : thick;
    // full Stokes: a ray deeper than tau_thick is in local equilibrium well
    // inside it, so its IQUV pass starts at tau_eq = 30 from the equilibrium
    // state x = K^-1 eps of the transfer matrix there (see start_iquv): the
    // part of the ray that start leaves out differs from equilibrium only by
    // the gradients of the source function, attenuated by exp(-(1 - p) 30)
    X.eq_start = (req->P.full && X.tau_thick < INFINITY && kTauEq < X.tau_thick) ? 1 : 0;
    X.tau_eq = X.eq_start ? kTauEq : X.tau_thick;
    X.tau_eq_f = (float)X.tau_eq;
    X.eq_min = X.eq_start ? std::min(kTauEqMin, X.tau_thick) : X.tau_thick;
  }
  if (m.v_kind == JSH_V_CONST_FLAT) {
    // getG, getD, get_n_los_prime (src/utils.cpp:147-162) in FP64
    double g = m.vp[0];
    double v = JSH_C * sqrt(1. - 1. / (g * g));
    double beta = v / JSH_C;
    double gamma = sqrt(1. / (1. - beta * beta));
    double D = 1. / (gamma * (1. - beta * nz));
    double f = (D + 1.) * (gamma / (gamma + 1.));
    X.v_const = 1;
    X.helical_bk = (m.b_kind == JSH_B_HELICAL_CONICAL && m.n_kind == JSH_N_BK && m.rnd_kind == JSH_RND_NONE) ? 1 : 0;
    const double n0p = m.n_plasma ? m.np[0] : m.np[0] / gamma;
    X.helical_log = (X.helical_bk && m.b_plasma && m.bp[0] != 0.0 && n0p > 0.0) ? 1 : 0;
    if (X.helical_log) {
      X.l2_b0 = (float)log2(fabs(m.bp[0]));
      X.l2_b0D = (float)log2(fabs(m.bp[0]) * D);
      X.l2_n0 = (float)log2(n0p);
      X.pk_h = (float)((s + 1.) / 2.);
      X.b_sign = m.bp[0] > 0.0 ? 1.f : -1.f;
      // the least of each factor between 2^-20 and 2^20 pc
      const double n_min = X.l2_n0 - 20.0 * fabs(m.np[1]), b_min = X.l2_b0 - 20.0 * fabs(m.bp[1]);
      const double w_min = std::min(0.0, X.l2_b0D - 20.0 * fabs(m.bp[1]) - 8.0);
      X.normal_range = (std::min(std::min(n_min, b_min), std::max(1.0, (s + 2.) / 2.) * w_min) > -126.0) ? 1 : 0;
    }
    X.D = (float)D;
    X.gamma = (float)gamma;
    X.beta = (float)beta;
    X.nlp[0] = (float)(D * nx);
    X.nlp[1] = (float)(D * ny);
    X.nlp[2] = (float)(D * nz - f * beta);
  }
  const double cb = JSH_Q_E / (2. * JSH_PI * JSH_M_E * JSH_C);  // nu_B per gauss
  const double cp = JSH_Q_E * JSH_Q_E / (JSH_PI * JSH_M_E);     // nu_p^2 per cm^-3
  const double fki = m.b_scalar ? m.fk_i * m.rnd_k : m.fk_i;
  const double fei = m.b_scalar ? m.fe_i * m.rnd_e : m.fe_i;
  for (int i = 0; i < req->n_nu; ++i) {
    double nu = nu_host[i];
    double Ak = JSH_PI * cp * pow(cb, (s + 2.) / 2.) * fki / (JSH_C * pow(nu, (s + 4.) / 2.));
    double Ae = JSH_PI * cp * pow(cb, (s + 1.) / 2.) * JSH_M_E * fei / (JSH_C * pow(nu, (s - 1.) / 2.));
    double Av = JSH_PI * cp * pow(cb, (s + 3.) / 2.) * m.fk_v / (JSH_C * pow(nu, (s + 5.) / 2.));
    double Aev = JSH_PI * cp * pow(cb, 1. + s / 2.) * JSH_M_E * m.fe_v / (JSH_C * pow(nu, s / 2.));
    double Af = 2. * JSH_PI * cp * cb / (JSH_C * nu * nu) * (m.kfr_factor + m.thermal_fraction);
    double Ac = JSH_PI * cp * cb * cb / (JSH_C * nu * nu * nu);
    double Gnu = pow(cb / nu, (s - 2.) / 2.);
    // scale: the source function at w = 1, D = 1
    double S = exp2(nearbyint(log2(Ae / Ak)));
    JshFreqConst& F = fc[i];
    F.ak = (float)(Ak * JSH_PC);
    F.ae = (float)(Ae * JSH_PC / S);
    F.av = (float)(Av * JSH_PC);
    F.aev = (float)(Aev * JSH_PC / S);
    F.af = (float)(Af * JSH_PC);
    F.ac = (float)(Ac * JSH_PC);
    F.c1 = (float)(m.kcr_a * m.kcr_b + m.thermal_fraction);
    F.c2 = (float)(m.kcr_a * Gnu);
    F.scale = S;
    F.atol = (float)(req->P.atol / S);
    F.r_kv = (float)((Av * JSH_PC) / (Ae * JSH_PC / S));
    F.r_ev = (float)((Aev * JSH_PC / S) / (Ak * JSH_PC));
    F.r_kc = (float)((Ac * JSH_PC) * (m.kcr_a * Gnu) / (Ak * JSH_PC));
    if (F.atol == 0.f && req->P.atol > 0.0) F.atol = FLT_MIN;  // below FP32 range: the smallest normal
    const float vals[9] = {F.ak, F.ae, F.av, F.aev, F.af, F.ac, F.r_kv, F.r_ev, F.r_kc};
    for (float x : vals) {
      if (!isfinite(x) || (x != 0.f && fabsf(x) < 1e-30f)) {
        jsh_set_error("frequency %g Hz puts the mixed-precision coefficients outside FP32 range; use FP64", nu);
        return JSH_ERR_INVALID;
      }
    }
  }
  return JSH_OK;
}
#endif  // !JSH_FARADAY_THICK_BUILD
