// jsh_autotune.cpp -- launch-shape search of the persistent schedule.
//
// The persistent transfer kernel's speed depends on four knobs that leave
// its results unchanged (an item's arithmetic does not depend on which lane
// or CTA runs it): the kernel build (default, or with capped registers for
// more resident warps), threads per CTA, resident CTAs per SM and the refill
// threshold (idle lanes of a warp before it pulls new items from the global
// queue).  The search times the caller's request under each shape with CUDA
// events on the context stream: first the context's present shape, which stays
// unless another one is faster, then a sweep over (build, block size, CTAs
// per SM, up to what fits of the kernels that the request runs) at the current
// refill threshold, then a sweep of the refill threshold at the best triple, then serial against overlapped passes of
// the split form (the deep rays' IQUV pass beside the other rays' passes)
// at the best shape, and the best of them in turns with the present one.  The
// faster of these becomes the context default, used
// by every later request whose params leave the knobs at 0.
//
// No counterpart in the reference, which renders on the CPU with an OpenMP
// loop over pixels (src/Observation.cpp:44-48).
#include <algorithm>
#include <vector>

#include "jsh_context.h"

namespace {

struct Timer {
  cudaEvent_t a = nullptr, b = nullptr;
  ~Timer() {
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
  }
};

// Time one run of the request with launch shape (bs, per_sm, refill) of the
// default or the register-capped (compact) kernel build.
int time_shape(jsh_ctx* ctx, Timer& T, const jsh_model_desc* model, const jsh_plane_desc* plane,
               const double* nu_hz, int32_t n_nu, jsh_params p, int bs, int per_sm, int refill, bool compact,
               double* ms) {
  p.block_size = bs;
  p.ctas_per_sm = per_sm;
  p.refill_threshold = refill;
  if (compact) p.flags |= JSH_FLAG_COMPACT_REGS;
  else p.flags &= ~JSH_FLAG_COMPACT_REGS;
  JSH_CUDA_TRY(cudaEventRecord(T.a, ctx->stream));
  int st = enqueue_single(ctx, model, plane, nu_hz, n_nu, &p, ctx->stream, nullptr, nullptr, nullptr);
  if (st) return st;
  JSH_CUDA_TRY(cudaEventRecord(T.b, ctx->stream));
  JSH_CUDA_TRY(cudaEventSynchronize(T.b));
  float f = 0.f;
  JSH_CUDA_TRY(cudaEventElapsedTime(&f, T.a, T.b));
  *ms = f;
  return JSH_OK;
}

}  // namespace

extern "C" int jsh_autotune(jsh_ctx* ctx, const jsh_model_desc* model, const jsh_plane_desc* plane,
                            const double* nu_hz, int32_t n_nu, const jsh_params* params, jsh_tuning* best) {
  if (!ctx || !model || !plane || !nu_hz || !params || !best) {
    jsh_set_error("null argument");
    return JSH_ERR_INVALID;
  }
  std::lock_guard<std::mutex> lk(ctx->mu);
  JSH_CUDA_TRY(cudaSetDevice(ctx->device));
  jsh_params p = *params;
  p.schedule = JSH_SCHED_PERSISTENT;
  // the shape sweeps time serial chains; overlap is tried last
  p.flags = (p.flags | JSH_FLAG_SERIAL_PASSES) & ~JSH_FLAG_OVERLAP_PASSES;
  Timer T;
  JSH_CUDA_TRY(cudaEventCreate(&T.a));
  JSH_CUDA_TRY(cudaEventCreate(&T.b));

  // warm-up run at the current default shape (first-touch of the workspace,
  // module load), then its time: the search starts from it
  struct Candidate {
    int bs, sm, rf;
    bool cp, ov;
    double ms;
  };
  const JshLaunchShape cur = ctx->shape;
  struct Restore {  // a candidate's knobs are all that its render has
    jsh_ctx* ctx;
    JshLaunchShape shape;
    ~Restore() { ctx->shape = shape; }
  } tuned{ctx, cur};
  ctx->shape.compact = ctx->shape.ctas_per_sm = ctx->shape.overlap_key = 0;
  auto run = [&](Candidate& c) {
    jsh_params q = p;
    if (c.ov) q.flags = (q.flags & ~JSH_FLAG_SERIAL_PASSES) | JSH_FLAG_OVERLAP_PASSES;
    return time_shape(ctx, T, model, plane, nu_hz, n_nu, q, c.bs, c.sm, c.rf, c.cp, &c.ms);
  };
  const uint64_t items = (uint64_t)plane->n_across * (uint64_t)plane->n_along * (uint64_t)n_nu;
  JshLaunchShape shape = jsh_params_shape(cur, &p);
  jsh_params overlapped = p;
  overlapped.flags = (p.flags & ~JSH_FLAG_SERIAL_PASSES) | JSH_FLAG_OVERLAP_PASSES;
  const bool may_overlap = jsh_overlap_passes(&overlapped, shape, items);
  Candidate start{cur.block_size, cur.ctas_per_sm, cur.refill_threshold, cur.compact != 0,
                  cur.overlap_key > 0 && may_overlap, 0.0};
  int st = run(start);
  if (!st) st = run(start);
  if (st) return st;
  Candidate best_c = start;
  auto keep = [&](const Candidate& c) {
    if (c.ms < best_c.ms) best_c = c;
  };

  // the kernels that this request runs (the render above has checked it)
  const bool full = p.output == JSH_OUT_FULL, mixed = p.precision == JSH_PREC_MIXED;
  JshRequest req;
  if (mixed) {
    uint64_t npix = 0;
    std::vector<JshFreqConst> fc((size_t)n_nu);
    st = jsh_prepare_request(ctx, model, plane, &p, n_nu, &req, &npix);
    if (!st) st = jsh_prepare_mixed(&req, nu_hz, fc.data());
    if (st) return st;
    shape.fused = jsh_fused_family(req.mix, p.flags) ? 1 : 0;
  }
  auto capped_law = [&](int bs) { return mixed && jsh_capped_law(req.mix, shape.single != 0, bs); };
  auto occupancy = [&](int bs, bool cp) {
    shape.compact = cp || capped_law(bs) ? 1 : 0;
    return jsh_persistent_occupancy(p.precision, full, bs, shape, items, ctx->num_sms);
  };
  // the register-capped builds: the mixed every-law and single-kernel ones
  const bool capped = mixed && (!shape.fused || shape.single);
  for (bool cp : {false, true}) {
    if (cp && !capped) continue;
    for (int bs : {64, 96, 128, 192, 256}) {
      const int occ = occupancy(bs, cp);
      if (occ < 1 || (cp && capped_law(bs))) continue;
      std::vector<int> per_sm = {occ};
      if (occ > 1) per_sm.push_back(occ - 1);
      if (occ > 2) per_sm.push_back(1);
      for (int k : per_sm) {
        Candidate c{bs, k, cur.refill_threshold, cp, false, 0.0};
        st = run(c);
        if (st) return st;
        keep(c);
      }
    }
  }
  const Candidate swept = best_c;
  for (int rf : {1, 2, 4, 8, 12, 16, 24, 32}) {
    Candidate c = swept;
    c.rf = rf;
    c.ov = false;
    if (rf == swept.rf && !swept.ov) continue;
    st = run(c);
    if (st) return st;
    keep(c);
  }
  // serial or overlapped passes (split form of the mixed schedule, requests
  // large enough to overlap); the sweeps above ran serial chains
  if (may_overlap && !best_c.ov) {
    Candidate c = best_c;
    c.ov = true;
    st = run(c);
    if (st) return st;
    keep(c);
  }
  // The best of ~40 single runs is partly luck: it replaces the start only if
  // it is faster in turns with it, by the best of three each.
  const bool moved = best_c.bs != start.bs || best_c.sm != start.sm || best_c.rf != start.rf ||
                     best_c.cp != start.cp || best_c.ov != start.ov;
  if (moved) {
    for (int k = 0; k < 3; ++k)
      for (Candidate* c : {&start, &best_c}) {
        Candidate again = *c;
        st = run(again);
        if (st) return st;
        c->ms = k == 0 ? again.ms : std::min(c->ms, again.ms);
      }
    if (!(best_c.ms < start.ms)) best_c = start;
  }
  const int b_bs = best_c.bs, b_rf = best_c.rf;
  const bool b_cp = best_c.cp, b_ov = best_c.ov;
  const double b_ms = best_c.ms;
  // all the CTAs that fit is the default of every kernel: another one's number may differ
  const int occ = occupancy(b_bs, b_cp);
  const int b_sm = best_c.sm > 0 ? best_c.sm : std::max(occ, 1);
  tuned.shape.block_size = b_bs;
  tuned.shape.ctas_per_sm = b_sm == occ ? 0 : b_sm;
  tuned.shape.refill_threshold = b_rf;
  tuned.shape.compact = b_cp ? 1 : 0;
  tuned.shape.overlap_key = b_ov ? JSH_OVERLAP_KEY : 0;
  best->block_size = b_bs;
  best->ctas_per_sm = b_sm;
  best->refill_threshold = b_rf;
  best->compact = b_cp ? 1 : 0;
  best->overlap = b_ov ? 1 : 0;
  best->ms = b_ms;
  return JSH_OK;
}
