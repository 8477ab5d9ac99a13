// jsh_launch.h -- host-callable launchers of the device kernels.  A batch is
// an array of JshRequest in device memory; every launcher enqueues on
// `stream` and returns the cudaError_t of the launch.
#pragma once

#include <cuda_runtime.h>

#include "jsh_request.h"

#define JSH_MAX_BATCH 64
// Deep-prefix bucket of overlapped passes (estimated optical depth of a ray
// at the request's first frequency >= 8), and the smallest request (work
// items) that overlaps them.
#define JSH_OVERLAP_KEY 43
#define JSH_OVERLAP_MIN_ITEMS 65536

// The initial values are every entry point's default (a context's may be tuned).
struct JshLaunchShape {
  int block_size = 128;  // threads per CTA of the transfer kernel
  int ctas_per_sm = 0;   // persistent schedule: CTAs per SM (0: occupancy max)
  // persistent schedule: refill when >= this many lanes idle.  A start is a
  // divergent stretch of code that the other lanes wait for (the IQUV kernel of
  // 705 176 items: 1.58 ms at 1, 1.43 at 8, 1.37 at 12, 1.38 at 16), and a group
  // of lanes is refilled with a second one.
  int refill_threshold = 12;
  int compact = 0;       // mixed persistent schedule: the register-capped build (<= 128 threads)
  int single = 0;        // mixed persistent schedule: tau and IQUV passes in one kernel (else split)
  int fused = 0;         // split form: every request of the batch is of the fused benchmark
                         // family (jsh_fused_family): launch the kernels built for it alone
  // mixed persistent schedule, optional: four events recorded on the stream
  // before the tau kernel, after it, after the IQUV ranking and after the
  // IQUV kernel (the single-kernel form records only the last two;
  // with overlapped passes: before the deep prefix's tau kernel, after the
  // other rays' tau kernel and IQUV ranking, and after both IQUV kernels)
  cudaEvent_t* marks = nullptr;
  // split form, optional: overlapped passes.  Rays whose rank bucket is at
  // least overlap_key (estimated optical depth >= 2^(overlap_key - 40)) form
  // the deep prefix: its tau pass runs first and its IQUV pass, which holds
  // the render's longest items, runs on `stream` at high priority while the
  // other rays' tau and IQUV passes run on `side` (fork[0] / fork[1]: events
  // of the fork and the join).  0 or no side stream: one serial chain.
  int overlap_key = 0;
  cudaStream_t side = nullptr;
  cudaEvent_t* fork = nullptr;
  // mixed precision, a launch on one request: its constants on the host (null:
  // the kernels read them from the record)
  const JshMixed* mix = nullptr;
  // mixed precision, full Stokes: run the kernels built with the
  // Faraday-thick mode (JSH_FLAG_FARADAY_THICK)
  int faraday_thick = 0;
};

// Ray generation: along sizes and centres (the sequential recurrences of
// pyLogspace / partial_sum, unless every request came with them: host_tables),
// then the across table.  max_along is the largest n_along of the batch.
cudaError_t jsh_launch_plane(const JshRequest* d_reqs, int n_req, uint64_t max_along, cudaStream_t stream,
                             bool host_tables = false);

// Zero `bytes` (a multiple of 16, 16-byte aligned) at p.
cudaError_t jsh_launch_clear(void* p, size_t bytes, cudaStream_t stream);

// Fills the record's cone_ray from its model and plane.
void jsh_prepare_hit(JshRequest* req);

// Hit every pixel's ray against the request's geometry, append the hit rays
// to req.hits (count in *req.n_hit, zeroed beforehand), write the outputs of
// missing pixels (zeros and geometry status) for every frequency.
cudaError_t jsh_launch_hit(const JshRequest* d_reqs, int n_req, uint64_t max_pix, cudaStream_t stream);

// Transfer every (hit ray, frequency) of the batch.  `queue` is a zeroed
// device counter used by the persistent schedule; max_items bounds the
// total work items (sum of npix * n_nu) for the static grid, max_hits the
// hit rays of one request.
cudaError_t jsh_launch_transfer(const JshRequest* d_reqs, int n_req, int precision, int schedule, bool full,
                                uint64_t max_items, uint64_t max_hits, const JshLaunchShape& shape,
                                unsigned int* queue, int num_sms, cudaStream_t stream);

// Hit arbitrary rays (origins/directions device arrays, directions already
// normalised on the device by this kernel as Ray::Ray does).
cudaError_t jsh_launch_hit_rays(const JshModel& model, const double* d_orig, const double* d_dir, int64_t n,
                                int32_t* d_nseg, double* d_seg, uint32_t* d_status, cudaStream_t stream);

// Ray origins of one compiled plane whose along/across tables are filled.
cudaError_t jsh_launch_plane_rays(const JshPlane& plane, double* d_orig, cudaStream_t stream);

// Gridded field interpolation at (z, r) points.
cudaError_t jsh_launch_grid_interp(const JshGrid& grid, int field, const double* d_zr, int64_t n,
                                   double nan_value, double* d_out, cudaStream_t stream);

// Largest resident CTAs per SM of block_size threads of the persistent transfer
// kernel that a request of at most `items` work items runs with `shape` (mixed:
// the IQUV kernel of the split form in the build of its law, its compact and its
// Faraday-thick build, or the single-kernel form; 0 if it cannot run them).
int jsh_persistent_occupancy(int precision, bool full, int block_size, const JshLaunchShape& shape, uint64_t items,
                             int num_sms);

// Nearest cell of n points (cm) of an uploaded cell set (checks), and the
// random unit directions of n counters (k0, k1, k2) of `seed`.
cudaError_t jsh_launch_cells_nearest(const JshCells& cells, const double* d_pts, int64_t n, int32_t* d_out,
                                     cudaStream_t stream);
cudaError_t jsh_launch_random_directions(uint64_t seed, const uint32_t* d_keys, int64_t n, double* d_out,
                                         cudaStream_t stream);
