// jsh_fp64.cu -- the all-FP64 transfer kernels: one group of five lanes per
// work item (static schedule, the plain GPU drop-in) and item-granular
// dynamic scheduling from a global queue.
#include <cuda_runtime.h>

#include "jsh_batch.cuh"
#include "jsh_launch.h"
#include "jsh_transfer64.cuh"

using namespace jsh;

namespace {

constexpr int kThreads64 = 128;
constexpr int kItemsPerCta = kThreads64 / 32 * kGroupsPerWarp;

// One item by the lanes of a group; lane 0 writes it.  Returns its counters
// (lane 0) and status.
__device__ __forceinline__ uint32_t run_item64(const JshRequest& R, unsigned long long local, const Group64& G,
                                               Ctl64& tot) {
  const unsigned nhit = *R.n_hit;
  const int f = (int)(local / nhit);
  const JshHit& H = R.hits[(unsigned)(local % nhit)];
  ItemOut o;
  if (R.P.full) transfer_item64<true>(R.model, R.plane, R.P, H, R.nu[f], f, G, o, tot);
  else transfer_item64<false>(R.model, R.plane, R.P, H, R.nu[f], f, G, o, tot);
  if (R.P.flags & JSH_FLAG_COST_MAP) o.l = (double)tot.evals;
  if (G.sub == 0) write_item(R, f, H.pix, o);
  return o.status;
}

// One lane group per (request, hit ray, frequency), all FP64.  Items are laid
// out frequency-major within a request so adjacent groups trace adjacent
// pixels (similar path lengths, less divergence).
__global__ void __launch_bounds__(kThreads64) transfer_static64_kernel(const JshRequest* __restrict__ reqs, int n_req) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  __shared__ double sh[kThreads64 / 32][kGroupsPerWarp * kGroup * NCOEF];
  batch_prefix(reqs, n_req, base);
  const Group64 G = group_of(sh[threadIdx.x / 32]);
  const unsigned long long w =
      (unsigned long long)blockIdx.x * kItemsPerCta + (threadIdx.x / 32) * kGroupsPerWarp + G.base / kGroup;
  const bool active = G.mask != 0 && w < base[n_req];
  int r = 0;
  Ctl64 tot{0, 0, 0, 0, 0, 0, 0};
  uint32_t status = 0;
  if (active) {
    r = find_request(base, n_req, w);
    status = run_item64(reqs[r], w - base[r], G, tot);
  }
  __syncwarp();
  add_counters(reqs, r, active && G.sub == 0, tot.evals, tot.acc, tot.rej, status);
}

// FP64 items with dynamic (queue) scheduling at item granularity.
__global__ void __launch_bounds__(kThreads64) transfer_queue64_kernel(const JshRequest* __restrict__ reqs, int n_req,
                                                                        unsigned long long* queue) {
  __shared__ unsigned long long base[JSH_MAX_BATCH + 1];
  __shared__ double sh[kThreads64 / 32][kGroupsPerWarp * kGroup * NCOEF];
  batch_prefix(reqs, n_req, base);
  const unsigned long long total = base[n_req];
  const Group64 G = group_of(sh[threadIdx.x / 32]);
  if (G.mask == 0) return;
  for (;;) {
    unsigned long long w = 0;
    if (G.sub == 0) w = atomicAdd(queue, 1ull);
    w = __shfl_sync(G.mask, w, G.base);
    if (w >= total) break;
    const int r = find_request(base, n_req, w);
    Ctl64 tot{0, 0, 0, 0, 0, 0, 0};
    const uint32_t status = run_item64(reqs[r], w - base[r], G, tot);
    if (G.sub == 0) {
      unsigned long long* c = reqs[r].counters;
      atomicAdd(&c[0], (unsigned long long)tot.evals);
      atomicAdd(&c[1], (unsigned long long)tot.acc);
      atomicAdd(&c[2], (unsigned long long)tot.rej);
      atomicOr(&c[3], (unsigned long long)status);
    }
  }
}

}  // namespace

cudaError_t jsh_launch_transfer_static64(const JshRequest* d_reqs, int n_req, uint64_t max_items, cudaStream_t stream) {
  const uint64_t blocks = (max_items + kItemsPerCta - 1) / kItemsPerCta;
  transfer_static64_kernel<<<(unsigned)blocks, kThreads64, 0, stream>>>(d_reqs, n_req);
  return cudaGetLastError();
}

cudaError_t jsh_launch_transfer_persistent64(const JshRequest* d_reqs, int n_req, uint64_t max_items,
                                             const JshLaunchShape& shape, unsigned int* queue, int num_sms,
                                             cudaStream_t stream) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, transfer_queue64_kernel, kThreads64, 0);
  if (per_sm < 1) per_sm = 1;
  unsigned blocks = (unsigned)(num_sms * per_sm);
  uint64_t need = (max_items + kItemsPerCta - 1) / kItemsPerCta;
  if (blocks > need) blocks = (unsigned)(need ? need : 1);
  transfer_queue64_kernel<<<blocks, kThreads64, 0, stream>>>(d_reqs, n_req, (unsigned long long*)queue);
  return cudaGetLastError();
}

int jsh_queue64_occupancy(int block_size) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, transfer_queue64_kernel, block_size, 0);
  return n;
}


