// fake_runtime.cpp -- jsh_capi.cpp on a fake CUDA runtime, on the CPU: device
// memory is host memory, copies happen at once, and every launch is an
// operation that a stream is behind of.  A fake transfer launch can fail.
// Scenarios (argv[1]) print one line per check and return 1 on a failed one.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>

#include "jsh_context.h"

namespace {
using Ops = std::set<int>;
std::map<void*, Ops> streams, events;
int n_ops = 0;
bool fail_transfer = false;
size_t device_bytes = 0, device_limit = (size_t)-1;
int n_mallocs = 0, last_single = -1;
std::map<void*, size_t> sizes;
int failed = 0;

void op(cudaStream_t s) { streams[(void*)s].insert(n_ops++); }
void check(bool ok, const char* what) {
  printf("%s: %s\n", ok ? "ok" : "FAILED", what);
  if (!ok) failed = 1;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  memset(p, 0, sizeof(*p));
  p->major = 10, p->minor = 3, p->multiProcessorCount = 152;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = *t = (size_t)64 << 30, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  ++n_mallocs;
  if (device_bytes + n > device_limit) return cudaErrorMemoryAllocation;
  *p = aligned_alloc(256, (n + 255) / 256 * 256);
  memset(*p, 0xcd, n);
  sizes[*p] = n;
  device_bytes += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  device_bytes -= sizes[p];
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)malloc(1), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free((void*)s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  for (int o : events[(void*)e]) streams[(void*)s].insert(o);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)malloc(1), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free((void*)e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  events[(void*)e] = streams[(void*)s];
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  op(st);
  return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  op(st);
  return memset(d, v, n), cudaSuccess;
}
}

// the library's kernels and the halves of the context that other files hold
int jsh_resolve_hull(jsh_ctx*, JshModel*) { return JSH_OK; }
int jsh_resolve_cells(jsh_ctx*, JshModel*) { return JSH_OK; }
int jsh_prepare_mixed(JshRequest*, const double*, JshFreqConst*) { return JSH_OK; }
void jsh_prepare_hit(JshRequest*) {}
cudaError_t jsh_run_peaks(int, double*, double*, double*, cudaStream_t) { return cudaSuccess; }
cudaError_t jsh_launch_clear(void* p, size_t n, cudaStream_t s) { return cudaMemsetAsync(p, 0, n, s); }
cudaError_t jsh_launch_plane(const JshRequest*, int, uint64_t, cudaStream_t s, bool) { return op(s), cudaSuccess; }
cudaError_t jsh_launch_plane_rays(const JshPlane&, double*, cudaStream_t s) { return op(s), cudaSuccess; }
cudaError_t jsh_launch_hit_rays(const JshModel&, const double*, const double*, int64_t, int32_t*, double*, uint32_t*,
                                cudaStream_t s) {
  return op(s), cudaSuccess;
}
cudaError_t jsh_launch_hit(const JshRequest* r, int, uint64_t, cudaStream_t s) {
  op(s);
  *r->n_hit = 5;
  return cudaSuccess;
}
cudaError_t jsh_launch_transfer(const JshRequest* r, int, int, int, bool, uint64_t, uint64_t, const JshLaunchShape& h,
                                unsigned*, int, cudaStream_t s) {
  op(s);
  if (h.side) op(h.side);
  last_single = h.single;
  if (fail_transfer) return cudaErrorInvalidValue;
  if (h.side) {
    cudaEventRecord(h.fork[1], h.side);
    cudaStreamWaitEvent(s, h.fork[1], 0);
  }
  for (int k = 0; k < 4; ++k) r->counters[k] = 100 + k;
  return cudaSuccess;
}

namespace {

jsh_model_desc model() {
  jsh_model_desc m;
  memset(&m, 0, sizeof(m));
  m.geometry.kind = JSH_GEO_CONE;
  m.geometry.direction[2] = 1.0;
  m.geometry.angle = 0.05;
  m.geometry.big_scale = 1e20;
  m.bfield.kind = JSH_B_HELICAL_CONICAL;
  m.bfield.p[0] = 0.1, m.bfield.p[1] = 1.0, m.bfield.p[2] = 0.8;
  m.nfield.kind = JSH_N_BK;
  m.nfield.p[0] = 500.0, m.nfield.p[1] = 2.0;
  m.vfield.kind = JSH_V_CONST_FLAT;
  m.vfield.p[0] = 10.0;
  m.s = 2.5;
  m.gamma_min = 10.0;
  return m;
}
jsh_plane_desc plane(uint64_t across, uint64_t along) {
  jsh_plane_desc p;
  memset(&p, 0, sizeof(p));
  p.n_across = across, p.n_along = along;
  p.lg_pixel_size_start_cm = p.lg_pixel_size_stop_cm = 17.0;
  p.los_angle = 0.1;
  return p;
}
jsh_params mixed(uint32_t flags = 0) {
  jsh_params p;
  jsh_params_default(&p);
  p.precision = JSH_PREC_MIXED;
  p.schedule = JSH_SCHED_PERSISTENT;
  p.flags = flags;
  return p;
}

// A render whose transfer launch fails leaves kernels on its stream and, where
// the passes overlap, on the side stream: the next user of the workspace waits
// for all of them.
void error_path() {
  for (bool overlap : {false, true}) {
    jsh_ctx* c = nullptr;
    check(jsh_ctx_create(0, 0, &c) == JSH_OK, "context");
    cudaStream_t s;
    cudaStreamCreateWithFlags(&s, 0);
    const jsh_model_desc m = model();
    const jsh_plane_desc p = plane(512, 1024);
    const jsh_params P = mixed(overlap ? JSH_FLAG_OVERLAP_PASSES : 0);
    const double nu = 1e10;
    jsh_image img;
    memset(&img, 0, sizeof(img));
    n_ops = 0;
    fail_transfer = true;
    check(jsh_observation_run_device(c, &m, &p, &nu, 1, &P, (void*)s, &img) == JSH_ERR_CUDA, "the launch fails");
    fail_transfer = false;
    check(n_ops > 3 && (int)events[(void*)c->ws_ready].size() == n_ops, "the workspace is in use by all it enqueued");
    check(jsh_observation_run_device(c, &m, &p, &nu, 1, &P, (void*)s, &img) == JSH_OK, "the next render runs");
    check((int)events[(void*)c->ws_ready].size() == n_ops, "and marks its end");
    cudaStreamDestroy(s);
    jsh_ctx_destroy(c);
  }
}

// The statistics of the last render are its own, whatever has used the
// workspace since.
void statistics() {
  jsh_ctx* c = nullptr;
  check(jsh_ctx_create(0, 0, &c) == JSH_OK, "context");
  const jsh_model_desc m = model();
  const jsh_params P = mixed();
  const double nu[3] = {1e10, 2e10, 3e10};
  static double rays[3 * 64 * 96], dir[3 * 64 * 96], seg[12 * 64 * 96];
  for (int k = 0; k < 3 * 64 * 96; ++k) rays[k] = dir[k] = 1.0;
  jsh_image img;
  memset(&img, 0, sizeof(img));
  jsh_stats want, got;
  for (int other = 0; other < 4; ++other) {
    const jsh_plane_desc p = plane(16, 24), q = plane(64, 96);
    check(jsh_observation_run_device(c, &m, &p, nu, 3, &P, (void*)c->stream, &img) == JSH_OK, "render");
    if (other == 0) {
      check(jsh_last_stats(c, &want) == JSH_OK && want.rhs_evals == 100 && want.n_work_items == 15, "its statistics");
    } else {
      int st = JSH_OK;
      if (other == 1) st = jsh_plane_rays(c, &q, rays, dir, nullptr);
      if (other == 2) st = jsh_trace_plane(c, &m, &q, nullptr, seg, nullptr);
      if (other == 3) st = jsh_hit_rays(c, &m, rays, dir, 64 * 96, nullptr, seg, nullptr);
      check(st == JSH_OK && jsh_last_stats(c, &got) == JSH_OK && !memcmp(&want, &got, sizeof(got)), "the same after");
    }
  }
  jsh_ctx_destroy(c);
}

// A request goes without its FP32 segments where the budget or the device has no
// room for them, without another attempt at every call, and has them again when
// the budget has.
void short_memory() {
  const jsh_model_desc m = model();
  const jsh_plane_desc p = plane(96, 128);
  const jsh_params P = mixed();
  const double nu = 1e10;
  jsh_image img;
  memset(&img, 0, sizeof(img));
  const size_t segments = (size_t)96 * 128 * JSH_MAX_SEG * sizeof(JshSeg32);
  JshRequestLayout L;
  jsh_request_layout(96 * 128, 128, 96, 1, false, false, &L);
  for (bool device : {false, true}) {
    jsh_ctx* c = nullptr;
    const size_t room = L.total + segments / 2;
    check(jsh_ctx_create(0, device ? 0 : L.total + segments + 65536, &c) == JSH_OK, "context");
    if (device) device_limit = device_bytes + room;
    void* other = nullptr;  // another user of the budget
    if (!device) {            // so much that the request is refused altogether
      check(jsh_alloc_device(c, segments + L.total, &other) == JSH_OK, "most memory");
      check(jsh_observation_run_device(c, &m, &p, &nu, 1, &P, (void*)c->stream, &img) == JSH_ERR_OOM, "refused");
      jsh_free_device(c, other, segments + L.total);
    }
    if (!device) check(jsh_alloc_device(c, segments / 2 + 65536, &other) == JSH_OK, "other memory");
    for (int k = 0; k < 3; ++k) {
      check(jsh_observation_run_device(c, &m, &p, &nu, 1, &P, (void*)c->stream, &img) == JSH_OK, "render");
      check(last_single == 1, "without segments");
      if (k == 0) n_mallocs = 0;
    }
    check(n_mallocs == 0, "no further attempt");
    if (!device) {
      jsh_free_device(c, other, segments / 2 + 65536);
      check(jsh_observation_run_device(c, &m, &p, &nu, 1, &P, (void*)c->stream, &img) == JSH_OK, "render");
      check(last_single == 0, "with segments");
    }
    device_limit = (size_t)-1;
    jsh_ctx_destroy(c);
  }
}

}  // namespace

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  if (!strcmp(what, "error")) error_path();
  else if (!strcmp(what, "statistics")) statistics();
  else if (!strcmp(what, "memory")) short_memory();
  else return 2;
  return failed;
}
