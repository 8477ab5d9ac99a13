// jsh_stripe.cu -- stripe mode: Observation::run_stripe
// (src/Observation.cpp:310-347) with integrate_tau (src/Observation.cpp:55-123)
// and Image::getStripe (src/Image.cpp:31-41), the tau-only pass along half of
// the central row that the reference's image-size search runs.
//
// One warp per stripe pixel (row n_across / 2, columns n_along / 2 ..
// n_along - 1), all FP64: the geometry hit, then per intersection a
// constant-step classical RK4 over the const-step time range [0, L] with
// dt = L / n (odeint runge_kutta4 through make_const_step_time_range: it
// steps while (t + dt) - L <= DBL_EPSILON, t = step * dt), stopped at the
// first yielded state with tau >= tau_max, whose tau is kept and whose
// later intersections are dropped; otherwise the state after the last step.
// dtau/dt = k_I does not depend on tau, so the two middle stages share one
// evaluation, and the three evaluations of 32 consecutive steps are spread over
// the lanes; their increments are then added in the order of the steps (the
// sums round as the serial steps do).  A ray that misses keeps tau = 0.  With a thread
// per pixel the 300 serial evaluations of FP64 set the time: 6.91 ms for the
// 1 000 pixels of a 2 000-column stripe on 8 CTAs, 0.39 ms with a warp per
// pixel (and the plane's recurrence on the host); 10 000 pixels 8.8 -> 5.1 ms,
// whose 20 000 columns keep the recurrence on the device.
#include <cuda_runtime.h>
#include <float.h>

#include <cmath>
#include <mutex>

#include "jsh_context.h"
#include "jsh_geometry.cuh"
#include "jsh_launch.h"
#include "jsh_transfer64.cuh"

using namespace jsh;

namespace {

// dtau/dt at path coordinate t.
__device__ __forceinline__ double tau_rate(const JshModel& m, const Path64& P, double t) {
  double k[NCOEF];
  P.at<0>(m, t, k, 0);
  return k[CK_I];
}

constexpr int kStripeThreads = 128;

__global__ void __launch_bounds__(kStripeThreads) stripe_tau_kernel(const JshRequest* __restrict__ req, double nu,
                                                                   double* __restrict__ tau_out) {
  __shared__ double increments[kStripeThreads / 32][96];
  double* inc = increments[threadIdx.x / 32];
  const JshRequest& R = *req;
  const JshPlane& pl = R.plane;
  const uint64_t c0 = pl.n_along / 2;
  const uint64_t col = c0 + ((uint64_t)blockIdx.x * kStripeThreads + threadIdx.x) / 32;
  const int lane = (int)(threadIdx.x & 31u);
  if (col >= pl.n_along) return;
  Hits h;
  geo_hit(R.model, R.cone_ray, plane_origin(pl, pl.n_across / 2, col), mk(pl.dx, pl.dy, pl.dz), h);
  const D3 rd = d3(pl.dx, pl.dy, pl.dz);
  const D3 nl = rd * -1.;
  const int n = R.P.n;
  const double tau_max = R.P.tau_max;
  double bg = 0.0;
  for (int s = 0; s < h.n; ++s) {
    const D3 pin = d3(h.s[s].in.x, h.s[s].in.y, h.s[s].in.z);
    const D3 dd = d3(h.s[s].out.x, h.s[s].out.y, h.s[s].out.z) - pin;
    const double length = sq(ad(ad(ml(dd.x, dd.x), ml(dd.y, dd.y)), ml(dd.z, dd.z)));
    const double dt = length / n;
    const Path64 P = path64(R.model, pin, rd, nl, nu);
    double x = 0.0;
    bool found = (x >= tau_max);
    if (dt > 0.0) {
      const double w1 = ml(1.0 / 6.0, dt), w2 = ml(1.0 / 3.0, dt);
      for (int64_t first = 0; !found && first <= (int64_t)n + 1; first += 32) {
        const int64_t step = first + lane;
        const double t = ml((double)step, dt);
        // the steps of the range are a prefix of the lanes: t grows with the step
        const bool in = step <= (int64_t)n + 1 && sb(ad(t, dt), length) <= DBL_EPSILON;
        const int steps = __popc(__ballot_sync(0xffffffffu, in));
        // evaluation e of the 3 * steps: stage e % 3 of step e / 3
        __syncwarp();
        for (int e = lane; e < 3 * steps; e += 32) {
          const int k = e / 3, stage = e - 3 * k;
          const double tk = ml((double)(first + k), dt);
          const double te = stage == 0 ? tk : stage == 1 ? ad(tk, ml(0.5, dt)) : ad(tk, dt);
          inc[e] = ml(stage == 1 ? w2 : w1, tau_rate(R.model, P, te));
        }
        __syncwarp();
        for (int i = 0; i < steps && !found; ++i) {
          const double bi = inc[3 * i + 1];
          x = ad(ad(ad(ad(x, inc[3 * i]), bi), bi), inc[3 * i + 2]);
          found = (x >= tau_max);
        }
        if (steps < 32) break;
      }
    }
    bg += x;
    if (found) break;
  }
  if (lane == 0) tau_out[col - c0] = bg;
}

}  // namespace

extern "C" int jsh_observation_run_stripe(jsh_ctx* ctx, const jsh_model_desc* model, const jsh_plane_desc* plane,
                                          double nu_hz, int32_t n, double tau_max, double* tau_host) {
  if (!ctx || !model || !plane || !tau_host) {
    jsh_set_error("null argument");
    return JSH_ERR_INVALID;
  }
  if (n < 1 || !(tau_max > 0) || !(nu_hz > 0) || !std::isfinite(nu_hz)) {
    jsh_set_error("stripe needs n >= 1, tau_max > 0 and a finite frequency > 0");
    return JSH_ERR_INVALID;
  }
  jsh_params P;
  jsh_params_default(&P);
  P.n = n;
  P.tau_max = tau_max;
  std::lock_guard<std::mutex> lk(ctx->mu);
  JSH_CUDA_TRY(cudaSetDevice(ctx->device));
  JshRequest req;
  uint64_t npix = 0;
  int st = jsh_prepare_request(ctx, model, plane, &P, 1, &req, &npix);
  if (st) return st;
  const uint64_t count = plane->n_along - plane->n_along / 2;
  JshRequestLayout L;
  jsh_request_layout(npix, plane->n_along, plane->n_across, 1, false, false, &L);
  const size_t off_out = (L.total + 255) / 256 * 256;
  st = keep_stats(ctx);
  if (st) return st;
  st = ensure_workspace(ctx, off_out + sizeof(double) * count);
  if (st) return st;
  JSH_CUDA_TRY(cudaEventSynchronize(ctx->ws_ready));
  char* base = (char*)ctx->ws;
  jsh_bind_request(&req, base, L, false);
  cudaStream_t s = ctx->stream;
  JshStage* stage = nullptr;
  st = jsh_next_stage(ctx, L, &stage);
  if (st) return st;
  JshWorkspaceUse use(ctx, s);
  st = jsh_upload_request(stage, &req, L, base, nullptr, s);
  if (st) return st;
  const JshRequest* d_req = (const JshRequest*)(base + L.off_req);
  if (count > 0) {
    stripe_tau_kernel<<<(unsigned)((count * 32 + kStripeThreads - 1) / kStripeThreads), kStripeThreads, 0, s>>>(d_req, nu_hz, (double*)(base + off_out));
    JSH_CUDA_TRY(cudaGetLastError());
    JSH_CUDA_TRY(cudaMemcpyAsync(tau_host, base + off_out, sizeof(double) * count, cudaMemcpyDeviceToHost, s));
  }
  JSH_CUDA_TRY(use.end());
  JSH_CUDA_TRY(cudaStreamSynchronize(s));
  return JSH_OK;
}
