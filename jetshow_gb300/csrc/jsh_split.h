// jsh_split.h -- the mixed path's kernels shared between its translation
// units: ranking and tau kernels (jsh_tau.cu) and the static and
// single-kernel forms (jsh_forms.cu and, with the Faraday-thick mode,
// jsh_forms_ft.cu), for the launch sequences of jsh_persistent.cu.
#pragma once

#include <cuda_runtime.h>

#include "jsh_request.h"

// (requests, their number, queue, refill threshold, part); the tau kernel takes
// the constants of a single request besides.
using TauKernel = void (*)(const JshRequest*, int, unsigned long long*, int, int, const JshMixed);
using IquvKernel = void (*)(const JshRequest*, int, unsigned long long*, int, int);
using StaticKernel = void (*)(const JshRequest*, int);
using SingleKernel = void (*)(const JshRequest*, int, unsigned long long*, int);

// The tau kernel (fused: built for the log-domain family alone; otherwise for
// every law, with a lane or a group of lanes per item; one: for a launch on a
// single request), its threads and its dynamic shared memory.
struct TauLaunch {
  TauKernel kernel;
  int block;
  size_t smem;
};
TauLaunch jsh_tau_kernel(bool fused, bool groups, bool one);

// Heaviest-first order of every request's hit rays; deep_key as
// rank_prefix_kernel; seg32: all of them have their segments in FP32.
void jsh_launch_rank(const JshRequest* d_reqs, int n_req, uint64_t max_hits, int deep_key, bool seg32,
                     cudaStream_t stream);

// Heaviest-first order of the items the tau kernel handed on (max_items: the
// batch's bound, the same for each of its requests).
void jsh_launch_iquv_rank(const JshRequest* d_reqs, int n_req, uint64_t max_items, int num_sms, int part,
                          cudaStream_t stream);

StaticKernel jsh_static_kernel(bool full);
SingleKernel jsh_single_kernel(bool full, bool compact);
StaticKernel jsh_static_kernel_ft(bool full);
SingleKernel jsh_single_kernel_ft(bool full, bool compact);
