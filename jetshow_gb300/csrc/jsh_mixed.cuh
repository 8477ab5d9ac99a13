// jsh_mixed.cuh -- the mixed-precision transfer's lane machine: FP32 right-hand sides
// and Runge-Kutta stages; FP64 time, step size, accumulated optical depth
// and Faraday rotation angle.  One work item is a (request, hit ray,
// frequency); its tau pass (src/Observation.cpp:126-214; a quadrature here,
// adaptive Gauss-Kronrod panels) and I/IQUV pass (src/Observation.cpp:242-308,
// src/System.cpp:41-63; Dormand-Prince) run as a per-lane state machine that
// advances by one panel or one Dormand-Prince attempt per call, so that
//  * the static schedule runs one item per thread to completion, and
//  * the persistent schedule keeps every warp busy: lanes whose ray has
//    finished are refilled from a global work queue (warp ballot + popc
//    rank, one atomic per warp) while the other lanes keep stepping.
//
// The IQUV state is integrated in a frame rotating with the Faraday angle
// chi (dchi/dt = k_F): with (Q, U) = R(chi) (q, u) the k_F terms of the
// reference right-hand side cancel and
//   dI/dt = eta_I - k_I I - k_Q (c q - s u) - k_V V
//   dq/dt = -k_I q + c (eta_Q - k_Q I) - s k_C V
//   du/dt = -k_I u - s (eta_Q - k_Q I) - c k_C V
//   dV/dt = eta_V - k_I V - k_V I + k_C (s q + c u),   c, s = cos, sin chi.
// chi accumulates in FP64; each stage rotates by the FP32 increment.  The
// error norm adds |err_chi| * |P| as the polarised-intensity error of the
// rotation.  Intensities are scaled by a per-frequency power of two and
// lengths are in pc so the FP32 state stays well inside its range.
//
// A step's coefficients depend on the stage points alone, so they are
// evaluated before the stages: five instead of six (the last two stages share
// their point), the stage derivatives in registers and the stages unrolled.
// On the 512x1024 conical jet the render went from 2.76 to 2.25 ms by that, on
// its 102x333 image (set by the heaviest ray's chain of steps) from 1.29 to
// 0.99 ms, on a ParabaloidCone image with the Faraday-thick mode from 71 to 40
// ms.  There is one copy of the coefficient code in a step (a rolled loop over
// the points, the coefficients in shared memory), so that it fits the SM
// instruction caches even when the lanes of a warp are in different phases;
// Stokes I alone, a shorter step, holds its points unrolled in registers.
#pragma once

#include <float.h>
#include <math.h>

#include <type_traits>

#include "jsh_batch.cuh"
#include "jsh_fields.cuh"
#include "jsh_fields32.cuh"
#include "jsh_launch.h"
#include "jsh_quadrature.h"
#include "jsh_transfer64.cuh"

namespace jsh {

namespace {

constexpr uint8_t PH_IDLE = 0, PH_TAU = 1, PH_IQUV = 2;
// Which passes a lane machine runs: both (the static schedule and the
// single-kernel persistent form), the tau pass only (the split form's first
// kernel: an item that needs an I/IQUV pass is handed on as a JshIquvItem),
// or the I/IQUV pass only (the split form's second kernel).
constexpr int PASS_BOTH = 0, PASS_TAU = 1, PASS_IQUV = 2;
// Optical depth of the equilibrium start of full-Stokes IQUV passes.
// Measured with the oracle's coefficients against the integration from
// tau_max (scipy Radau at rtol 1e-11) on 27 rays of depth 94 .. 3.2e4 of the
// conical and ParabaloidCone jets at their lowest and highest frequencies:
// worst 2.2e-6 of I in I, Q, U, V at tau_eq = 30 (2.6e-5 at 20), against
// 3e-10 for the zero state at tau_thick = 89.
constexpr double kTauEq = 30.0;
// Smallest total depth of a ray started in equilibrium at kTauEq: behind the
// start lie at least 10 optical depths, so the state there is within
// exp(-(1 - p) 10) of equilibrium before the 30 depths in front attenuate it.
// The rays just shallower than this, integrated whole from their far end,
// are the render's longest items (their cost grows with their depth): on the
// 512x1024 conical jet lowering it from 50 to 40 took the longest from 4 585
// to 3 883 evaluations with the errors against the converged oracle of 300
// rays of depth 25 .. 80 unchanged (I 5.8e-6, Q 4.1e-6 of max I; 35 raised
// Q to 6.8e-6).
constexpr double kTauEqMin = 40.0;
constexpr double INV_PC = 1.0 / JSH_PC;
// First panel width of a tau-pass segment: a quarter of it (the panels then
// adapt; four panels of 15 nodes resolve the features of a segment that one
// panel's error estimate could miss).
constexpr float kPanelsPerSegment = 4.f;

// Tableau entry a_sj in FP32 (row 6 = the 5th-order weights b), folded to an
// immediate operand where s and j are compile-time constants.
__host__ __device__ constexpr float dp_a32(int s, int j) {
  return s == 1 ? (j == 0 ? (float)dp::A21 : 0.f)
       : s == 2 ? (j == 0 ? (float)dp::A31 : j == 1 ? (float)dp::A32 : 0.f)
       : s == 3 ? (j == 0 ? (float)dp::A41 : j == 1 ? (float)dp::A42 : j == 2 ? (float)dp::A43 : 0.f)
       : s == 4 ? (j == 0 ? (float)dp::A51 : j == 1 ? (float)dp::A52 : j == 2 ? (float)dp::A53
                  : j == 3 ? (float)dp::A54 : 0.f)
       : s == 5 ? (j == 0 ? (float)dp::A61 : j == 1 ? (float)dp::A62 : j == 2 ? (float)dp::A63
                  : j == 3 ? (float)dp::A64 : j == 4 ? (float)dp::A65 : 0.f)
       : s == 6 ? (j == 0 ? (float)dp::B1 : j == 2 ? (float)dp::B3 : j == 3 ? (float)dp::B4
                  : j == 4 ? (float)dp::B5 : j == 5 ? (float)dp::B6 : 0.f)
       : 0.f;
}

// Dormand-Prince nodes c, error weights e = b - b_hat and dense-output
// weights d in FP32.
__host__ __device__ constexpr float dp_c32(int s) {
  return s == 1 ? (float)dp::C2 : s == 2 ? (float)dp::C3 : s == 3 ? (float)dp::C4 : s == 4 ? (float)dp::C5
       : s >= 5 ? 1.f : 0.f;
}
__host__ __device__ constexpr float dp_e32(int j) {
  return j == 0 ? (float)dp::E1 : j == 2 ? (float)dp::E3 : j == 3 ? (float)dp::E4 : j == 4 ? (float)dp::E5
       : j == 5 ? (float)dp::E6 : j == 6 ? (float)dp::E7 : 0.f;
}
__constant__ float c_C[7] = {0, (float)dp::C2, (float)dp::C3, (float)dp::C4, (float)dp::C5, 1.f, 1.f};
__constant__ float c_E[7] = {(float)dp::E1, 0, (float)dp::E3, (float)dp::E4, (float)dp::E5, (float)dp::E6,
                             (float)dp::E7};
__constant__ float c_D[7] = {(float)dp::D1, 0, (float)dp::D3, (float)dp::D4, (float)dp::D5, (float)dp::D6,
                             (float)dp::D7};

// Compensated FP32 pair x = hi + lo, |lo| <= ulp(hi) / 2 (about 48 bits):
// the step-control state (segment coordinate, remainder, optical depth,
// Faraday angle, base point) is carried in these pairs because GB300 runs
// FP64 at 1/64 of the FP32 rate; the additions are error-free
// transformations (Knuth's two-sum, Dekker's product error by fma).
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF df_of(double x) {
  const float h = (float)x;
  return DF{h, (float)(x - (double)h)};
}
__device__ __forceinline__ double df_val(DF a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ DF df_norm(float s, float e) {
  const float hi = s + e;
  return DF{hi, e - (hi - s)};
}
// a + b
__device__ __forceinline__ DF df_add(DF a, float b) {
  const float s = a.hi + b;
  const float bb = s - a.hi;
  const float e = ((a.hi - (s - bb)) + (b - bb)) + a.lo;
  return df_norm(s, e);
}
// a - b
__device__ __forceinline__ DF df_sub(DF a, DF b) {
  const float s = a.hi - b.hi;
  const float bb = s - a.hi;
  const float e = ((a.hi - (s - bb)) - (b.hi + bb)) + (a.lo - b.lo);
  return df_norm(s, e);
}
// p + t * d rounded to FP32 (p, t, d pairs)
__device__ __forceinline__ float df_axpy_round(DF t, DF d, DF p) {
  const float m = t.hi * d.hi;
  const float me = fmaf(t.hi, d.hi, -m);  // exact product error
  const float s = p.hi + m;
  const float bb = s - p.hi;
  const float se = (p.hi - (s - bb)) + (m - bb);
  return s + (((se + me) + p.lo) + fmaf(t.hi, d.lo, t.lo * d.hi));
}

struct Lane {
  int r, f;
  uint32_t h;
  uint8_t phase;
  int8_t seg, nseg;
  int8_t first_seg;      // segment where the IQUV pass starts inside (-1: at its end)
  bool init;
  bool last;             // dt was truncated to reach the segment's end
  uint8_t ft;            // IQUV pass in the Faraday-thick mode (quasi-static polarisation)
  uint8_t ft_cool;       // steps before the Faraday-thick mode may be tried again
  uint8_t ft_back;       // entry estimates in a row that found the transient too large (back-off)
  DF p0x, p0y, p0z;      // segment start [pc]
  float bx, by, bz;      // p0 + t d rounded to FP32 after each accepted step:
                         // stage points are b + c h d in FP32 (error u |b|)
  DF length, t;          // segment length and coordinate [pc]
  float dt;              // [pc]
  DF tau_seg;            // optical depth of the current tau segment
  float thick_left;      // tau_thick - (depth of the finished segments)
  float first_div;       // I/IQUV pass: divisor of a segment's first step
  double tau_bg, thick;  // tau pass: depth and length of the finished segments
  double t_first;        // [pc] IQUV start on first_seg: tau_max crossing or optically thick point
  DF chi;                // Faraday rotation angle, kept reduced to [-pi, pi]
  float x[4];
  float k1[5];
  float s1;  // noise scale of k1
  float kI1; // k_I at the point of k1
  int32_t nsteps, fails;
  uint32_t status;
  uint32_t evals, acc, rej;
  uint32_t evals0;       // split form, IQUV kernel: the item's tau-pass evaluations (cost map)
  int32_t tri;           // gridded fields on one grid: triangle of the last evaluation (-1: none)
};

// Stage storage of this thread in shared memory, thread-major: t = shared +
// tid * stride, every access a fixed offset from one base register, and the
// odd stride maps a warp's 32 threads onto 32 distinct banks.  It holds the
// stages' k_I of a Dormand-Prince tau pass (7 words) or, in the kernels
// built for every field law, the coefficients of an I/IQUV step's stage
// points (StageWidth<FULL>::kWords).
template <bool FULL>
struct StageWidth {
  static constexpr int NK = FULL ? 5 : 1;        // stage components: the IQUV state and chi, or I only
  static constexpr int NX = FULL ? 4 : 1;
  static constexpr int NC = FULL ? 8 : 2;        // coefficients of a stage point
  static constexpr int kWords = FULL ? 49 : 13;  // six points, odd
};
constexpr int kTauWords = 17;  // the 15 nodes of a panel, odd

// Lanes that run one item: one, or a group of kGroupLanes.  A group's lanes
// hold the same state and take the same branches; each evaluates one stage
// point of a Dormand-Prince step (or every fifth node of a panel) and the
// results are exchanged, so a step costs one evaluation's latency instead of
// five.  Lane 0 writes the outputs.  The fused build has a copy of the step
// for each (NG = 1, 5), the builds for every field law one (NG = 0: the group's
// size is LaneGroup::n).

// The I/IQUV kernels' files are compiled twice: as is, and by the _ft.cu files with
// JSH_FARADAY_THICK_BUILD 1 for requests that ask for the Faraday-thick mode
// (JSH_FLAG_FARADAY_THICK).  The mode's bookkeeping in the step costs the
// other requests 15 to 33 % of the IQUV kernel even where it never engages
// (128x128: 75 -> 86 us; 512x1024 x 4: 1.15 -> 1.53 ms), so the default kernels
// are built without it.
#ifndef JSH_FARADAY_THICK_BUILD
#define JSH_FARADAY_THICK_BUILD 0
#endif
constexpr bool kFtm = JSH_FARADAY_THICK_BUILD != 0;
// fused I/IQUV step: five points of two float4 (three with the Faraday-thick
// mode), the groups spread over the banks
constexpr int kGroupWords = kFtm ? 76 : 52;
// the same of a lane: five points of two float4, the lanes over the banks
constexpr int kLaneWords = 44;

// acc = sum_{j < S} a_Sj K_j over the stage derivatives held in registers
// (S and j compile-time: the tableau entries are immediate operands).
template <int S, int NK>
__device__ __forceinline__ void combine_stage(const float (&K)[7][NK], float* acc) {
#pragma unroll
  for (int c = 0; c < NK; ++c) acc[c] = 0.f;
#pragma unroll
  for (int j = 0; j < S; ++j) {
#pragma unroll
    for (int c = 0; c < NK; ++c) acc[c] = fmaf(dp_a32(S, j), K[j][c], acc[c]);
  }
}

__device__ __forceinline__ double seg_len_cm(const JshHit& H, int s, double ox, double oy, double oz) {
  double dx = ox - H.seg[s][0], dy = oy - H.seg[s][1], dz = oz - H.seg[s][2];
  return sqrt((dx * dx + dy * dy) + dz * dz);
}

// auto_n of src/Observation.cpp:254-258: steps_schedule (src/utils.cpp:354-366,
// default limits 0.1 and 100) in FP32.  It only sets the first step guess of
// a segment, so FP32 rounding near an integer boundary changes no accuracy;
// in FP64 its log and pow were a large share of the per-item FP64 work
// (GB300 runs FP64 at 1/64 of the FP32 rate).
__device__ __forceinline__ float first_step_divisor(double tau_bg, int n) {
  if (!(tau_bg > 0.1)) return (float)n;
  if (tau_bg >= 100.0) return (float)(10 * n);
  const float b = 2.30258509f;                              // -log(0.1)
  const float k = (float)(10 * n) / ((4.60517019f + b) * (4.60517019f + b));  // log(100) + b
  const float l = logf((float)tau_bg) + b;
  return ceilf(fmaf(k * l, l, (float)n));
}

// Segment s of hit h: the hit kernel's record, or (ANY) computed here where the
// request has no memory for them, with the same rounding, so the same images.
// Such requests run in the static or the single-kernel form: the code costs the
// split form's fused IQUV kernel 4 registers and a quarter of its warps.
static __device__ __noinline__ void segment_of_hit(const JshHit& H, int s, JshSeg32* q) {
  const double* p = H.seg[s];
  *q = segment32(mk(p[0], p[1], p[2]), mk(p[3], p[4], p[5]));
}
template <bool ANY>
__device__ __forceinline__ std::conditional_t<ANY, JshSeg32, const JshSeg32&> segment_of(const JshRequest& R, uint32_t h,
                                                                                         int s) {
  if constexpr (ANY) {
    JshSeg32 q;
    if (R.seg32) return R.seg32[(uint64_t)h * JSH_MAX_SEG + s];
    segment_of_hit(R.hits[h], s, &q);
    return q;
  } else {
    return R.seg32[(uint64_t)h * JSH_MAX_SEG + s];
  }
}

__device__ __forceinline__ void start_segment(Lane& L, DF px, DF py, DF pz, DF len) {
  L.length = len;
  L.t = DF{0.f, 0.f};
  L.p0x = px;
  L.p0y = py;
  L.p0z = pz;
  L.bx = L.p0x.hi;
  L.by = L.p0y.hi;
  L.bz = L.p0z.hi;
  L.last = false;
  L.init = false;
  L.nsteps = 0;
  L.fails = 0;
}

// Total optical depth of the lane's tau pass, which is in its last segment.
__device__ __forceinline__ double tau_total(const Lane& L) {
  return L.seg == 0 ? df_val(L.tau_seg) : L.tau_bg + df_val(L.tau_seg);
}

template <int PASS>
__device__ __forceinline__ void begin_tau_segment(Lane& L, const JshRequest& R, const JshMixed& X) {
  const JshSeg32& S = segment_of<PASS == PASS_BOTH>(R, L.h, L.seg);
  start_segment(L, DF{S.in[0], S.in[1]}, DF{S.in[2], S.in[3]}, DF{S.in[4], S.in[5]}, DF{S.len[0], S.len[1]});
  const float len = L.length.hi + L.length.lo;
  if (L.seg == 0) {
    L.thick = S.len_cm;
    L.thick_left = X.tau_eq_f;
  } else {
    L.tau_bg = df_val(L.tau_seg);  // two segments at most: that of segment 0
    L.thick += S.len_cm;
    L.thick_left = (float)(X.tau_eq - L.tau_bg);
  }
  L.tau_seg = DF{0.f, 0.f};
  if (!X.helical_log) {
    // the Dormand-Prince tau pass: the reference's first step L / n
    L.dt = len / (float)R.P.n;
    return;
  }
  L.dt = len * (1.f / kPanelsPerSegment);
  // closest approach of the segment to the jet (z) axis, where the fields'
  // azimuthal direction turns fastest (a helical B flips within the
  // approach distance): a panel breakpoint when it lies inside the segment
  // and the approach distance is below 1/32 of the segment, finer than the
  // nodes of the first panels resolve (L.k1[2], [pc] along it; L.k1[3] the
  // approach distance, at least 1e-6 of the segment).  FP32 is enough: it
  // only places panels.
  const float ux = X.dhi[0], uy = X.dhi[1];
  const float uu = fmaf(ux, ux, uy * uy);
  L.k1[2] = INFINITY;
  L.k1[3] = 1e-6f * len;
  if (uu > 0.f) {
    const float sc = -fmaf(L.p0x.hi, ux, L.p0y.hi * uy) / uu;
    if (sc > 0.f && sc < len) {
      const float cx = fmaf(sc, ux, L.p0x.hi), cy = fmaf(sc, uy, L.p0y.hi);
      const float rmin = sqrtf(fmaf(cx, cx, cy * cy));
      if (rmin < len * (1.f / 32.f)) {
        L.k1[2] = sc;
        L.k1[3] = fmaxf(rmin, L.k1[3]);
      }
    }
  }
}

template <int PASS>
__device__ __forceinline__ void begin_iquv_segment(Lane& L, const JshRequest& R) {
  const int s = L.seg;
  if (s == L.first_seg) {
    // inside the segment, t_first from its near end
    L.first_seg = -1;
    const JshHit& H = R.hits[L.h];
    const double tc = L.t_first * JSH_PC;
    const double ox = H.seg[s][0] + R.plane.rx * tc, oy = H.seg[s][1] + R.plane.ry * tc,
                 oz = H.seg[s][2] + R.plane.rz * tc;
    start_segment(L, df_of(ox * INV_PC), df_of(oy * INV_PC), df_of(oz * INV_PC),
                  df_of(seg_len_cm(H, s, ox, oy, oz) * INV_PC));
  } else {
    const JshSeg32& S = segment_of<PASS == PASS_BOTH>(R, L.h, s);
    start_segment(L, DF{S.out[0], S.out[1]}, DF{S.out[2], S.out[3]}, DF{S.out[4], S.out[5]}, DF{S.len[0], S.len[1]});
  }
  L.dt = (L.length.hi + L.length.lo) / L.first_div;
  L.ft = 0;  // (Q, U) enters a segment as it left the last one, not quasi-static
  L.ft_cool = 0;
  L.ft_back = 0;
}

// Work item w of the batch.  Unranked: frequency-major over the hit list.
// Ranked (persistent schedule): all frequencies of a ray together, rays in
// the heaviest-first order of the ranking kernels; part 1 (the rays after
// the deep prefix of overlapped passes) starts after the deep prefix.
template <int PASS>
__device__ __forceinline__ void lane_start(Lane& L, const JshRequest* __restrict__ reqs,
                                           const unsigned long long* base, int n_req, unsigned long long w,
                                           bool ranked, int part = 0, const JshMixed* one = nullptr) {
  int r = find_request(base, n_req, w);
  const JshRequest& R = reqs[r];
  unsigned long long local = w - base[r];
  L.r = r;
  if (ranked) {
    const unsigned long long rank = local / (unsigned)R.n_nu;
    L.f = (int)(local - rank * (unsigned)R.n_nu);
    L.h = R.order[rank + (part ? R.buckets[JSH_RANK_DEEP] : 0u)];
  } else {
    unsigned nhit = *R.n_hit;
    L.f = (int)(local / nhit);
    L.h = (uint32_t)(local % nhit);
  }
  const JshHit& H = R.hits[L.h];
  L.phase = PH_TAU;
  L.seg = 0;
  L.nseg = (int8_t)H.nseg;
  L.first_seg = -1;
  L.tau_bg = 0.0;
  L.thick = 0.0;
  L.t_first = -1.0;
  L.chi = DF{0.f, 0.f};
  L.x[0] = L.x[1] = L.x[2] = L.x[3] = 0.f;
  L.status = (uint32_t)H.status | JSH_ST_HIT;
  L.evals = L.acc = L.rej = 0;
  L.tri = -1;
  L.ft = 0;
  L.ft_cool = 0;
  L.evals0 = 0;
  begin_tau_segment<PASS>(L, R, one ? *one : R.mix);
}

// Per-lane totals of a request's counters (right-hand-side evaluations,
// accepted and rejected steps, status OR) over the items the lane finished
// or handed on.  They reach the request's counters when the lane moves to an
// item of another request (per lane) and when the kernel ends (one atomic
// per warp and counter), instead of four atomics per item on the same four
// words: those kept one L2 slice's atomic unit busy for ~60 % of the tau
// kernel's time and set its length once its arithmetic shrank.
struct Tally {
  int r;
  unsigned long long evals;
  uint32_t acc, rej, status;
};

__device__ __forceinline__ Tally tally_new() { return Tally{-1, 0ull, 0u, 0u, 0u}; }

__device__ __forceinline__ void tally_add(Tally& T, const JshRequest* __restrict__ reqs, int r, uint32_t evals,
                                          uint32_t acc, uint32_t rej, uint32_t status) {
  if (r != T.r) {
    if (T.r >= 0) {
      unsigned long long* c = reqs[T.r].counters;
      atomicAdd(&c[0], T.evals);
      atomicAdd(&c[1], (unsigned long long)T.acc);
      atomicAdd(&c[2], (unsigned long long)T.rej);
      atomicOr(&c[3], (unsigned long long)T.status);
    }
    T = Tally{r, 0ull, 0u, 0u, 0u};
  }
  T.evals += evals;
  T.acc += acc;
  T.rej += rej;
  T.status |= status;
}

// Flush at the end of a kernel; every lane of the warp calls it.
__device__ __forceinline__ void tally_flush(const Tally& T, const JshRequest* __restrict__ reqs) {
  add_counters(reqs, T.r, T.r >= 0, T.evals, T.acc, T.rej, T.status);
}

// Writes one finished item (the Stokes vector rotated back to the lab frame
// in FP64); its counters go to the lane's tally.
__device__ __noinline__ void write_finished(const JshRequest* __restrict__ reqs, int r, int f, uint32_t h,
                                            double tau_bg, double thick, float chi_hi, float chi_lo, float x0,
                                            float x1, float x2, float x3, uint32_t status, uint32_t evals) {
  const JshRequest& R = reqs[r];
  const JshHit& H = R.hits[h];
  uint64_t q = (uint64_t)f * R.npix + (uint64_t)H.pix;
  double S = R.mix.fc[f].scale;
  // rotation by chi = hi + lo (|hi| <= pi): sin, cos of hi in FP32 and the
  // first-order correction for lo; (Q, U) need ~1e-7 of P, far above this
  float sh, ch;
  sincosf(chi_hi, &sh, &ch);
  const float ss = fmaf(chi_lo, ch, sh), sc = fmaf(-chi_lo, sh, ch);
  if (R.tau) R.tau[q] = tau_bg;
  if (R.l) R.l[q] = (R.P.flags & JSH_FLAG_COST_MAP) ? (double)evals : thick;
  if (R.I) R.I[q] = S * (double)x0;
  if (R.Q) R.Q[q] = S * (double)fmaf(sc, x1, -ss * x2);
  if (R.U) R.U[q] = S * (double)fmaf(ss, x1, sc * x2);
  if (R.V) R.V[q] = S * (double)x3;
  if (R.status) R.status[q] = status;
}

__device__ __forceinline__ void lane_finish(Lane& L, const JshRequest* __restrict__ reqs, Tally& T, bool lead) {
  L.phase = PH_IDLE;
  if (!lead) return;
  write_finished(reqs, L.r, L.f, L.h, L.tau_bg, L.thick, L.chi.hi, L.chi.lo, L.x[0], L.x[1], L.x[2], L.x[3],
                 L.status, L.evals);
  tally_add(T, reqs, L.r, L.evals, L.acc, L.rej, L.status);
}

// Split form, IQUV kernel: the item's Stokes planes and final status (its
// tau and l planes were written by the tau kernel; with the cost map, l is
// rewritten with the evaluations of both passes).
__device__ __noinline__ void write_finished_iquv(const JshRequest* __restrict__ reqs, int r, int f, uint32_t h,
                                                 float chi_hi, float chi_lo, float x0, float x1, float x2,
                                                 float x3, uint32_t status, uint32_t evals0, uint32_t evals) {
  const JshRequest& R = reqs[r];
  const JshHit& H = R.hits[h];
  uint64_t q = (uint64_t)f * R.npix + (uint64_t)H.pix;
  double S = R.mix.fc[f].scale;
  float sh, ch;
  sincosf(chi_hi, &sh, &ch);
  const float ss = fmaf(chi_lo, ch, sh), sc = fmaf(-chi_lo, sh, ch);
  if (R.l && (R.P.flags & JSH_FLAG_COST_MAP)) R.l[q] = (double)(evals0 + evals);
  if (R.I) R.I[q] = S * (double)x0;
  if (R.Q) R.Q[q] = S * (double)fmaf(sc, x1, -ss * x2);
  if (R.U) R.U[q] = S * (double)fmaf(ss, x1, sc * x2);
  if (R.V) R.V[q] = S * (double)x3;
  if (R.status) R.status[q] = status;
}

// Optical depth the I/IQUV pass of an item integrates through, bucketed by
// half octaves from 2^-19 up.  The pass's cost grows with it, also where the
// ray is thin (its Faraday depth grows with the optical depth: on a
// ParabaloidCone image the mean cost falls from 8 700 evaluations at depth 1
// to 430 at 2^-11), so the order puts the longest items first and items of one
// length into one warp.
__device__ __forceinline__ uint8_t iquv_cost_key(float tau, bool eq, bool first, const JshMixed& X) {
  float d = first ? fminf(tau, (float)X.tau_thick) : tau;
  // from the equilibrium at tau_eq the pass is the shorter the deeper the ray
  // (512x1024 conical jet: 1 450 evaluations at depth 50, 820 at 240, 425 at
  // 10^4, as rays of depth 30, 10 and 2)
  if (eq) d = (float)X.tau_eq * sqrtf((float)X.eq_min / tau);
  if (!(d > 0.f)) return 1;
  const int k = (int)floorf(2.f * __log2f(d)) + 40;
  return (uint8_t)min(max(k, 1), JSH_RANK_BUCKETS - 1);
}

// Split form, tau kernel: hand an item whose I/IQUV pass is still to run to
// the IQUV kernel.  Writes the item's l plane (and its tau plane, unless the
// depth is left a pair for the ranking kernel to convert) and its tau-pass
// counters, appends its record to the request's list of its part (one
// atomic per request among the lanes that emit together).
__device__ __noinline__ void emit_iquv(const JshRequest* __restrict__ reqs, int part, int r, int f, uint32_t h,
                                       bool pair, DF tau, double tau_bg, double thick, double t_first, int first_seg,
                                       int nseg, bool eq, uint32_t status, uint32_t evals) {
  const JshRequest& R = reqs[r];
  const JshHit& H = R.hits[h];
  uint64_t q = (uint64_t)f * R.npix + (uint64_t)H.pix;
  if (R.tau && !pair) R.tau[q] = tau_bg;
  if (R.l) R.l[q] = (R.P.flags & JSH_FLAG_COST_MAP) ? (double)evals : thick;
  const unsigned mask = __activemask();
  const unsigned peers = __match_any_sync(mask, r);
  const int leader = __ffs(peers) - 1;
  const unsigned lane = threadIdx.x & 31u;
  uint32_t slot = 0;
  if ((int)lane == leader) slot = atomicAdd(R.iq_count + part, (uint32_t)__popc(peers));
  slot = __shfl_sync(peers, slot, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
  if (part) slot += R.buckets[JSH_RANK_DEEP] * (uint32_t)R.n_nu;
  JshIquvItem it;
  it.h = h;
  it.f = (uint16_t)f;
  it.key = iquv_cost_key(pair ? tau.hi : (float)tau_bg, eq, first_seg >= 0, R.mix);
  it.flags = (uint8_t)((nseg & 3) | (eq ? 4 : 0) | ((first_seg + 1) << 3) | (pair ? 32 : 0));
  it.status = status;
  it.evals = evals;
  if (pair) {
    it.tau_pair[0] = tau.hi;
    it.tau_pair[1] = tau.lo;
  } else {
    it.tau_bg = tau_bg;
  }
  it.t_first = t_first;
  R.iq_items[slot] = it;
}

// Bisection for the tau_max crossing on the dense output of the last
// Dormand-Prince step (src/Observation.cpp:166-190); returns the crossing
// time [pc], or -1 without convergence.
__device__ __noinline__ double crossing_time(double tau_old, double t_old, double dt_used, float h, float k1,
                                             float k3, float k4, float k5, float k6, float k7, float inc,
                                             double tau_max, double tau_prec) {
  const float ydiff = inc;
  const float bspl = h * k1 - ydiff;
  const float r4 = ydiff - h * k7 - bspl;
  const float r5 = h * (c_D[0] * k1 + c_D[2] * k3 + c_D[3] * k4 + c_D[4] * k5 + c_D[5] * k6 + c_D[6] * k7);
  double t0 = t_old, t1 = t_old + dt_used, xm = tau_old + (double)inc, tm;
  int it = 0;
  while (fabs(xm - tau_max) > tau_prec) {
    if (++it > 200) return -1.0;
    tm = 0.5 * (t0 + t1);
    float th = (float)((tm - t_old) / dt_used), th1 = 1.f - th;
    xm = tau_old + (double)(th * (ydiff + th1 * (bspl + th * (r4 + th1 * r5))));
    if (xm > tau_max) t1 = tm;
    else t0 = tm;
  }
  return 0.5 * (t0 + t1);
}

// Stokes derivatives of the I/IQUV pass from the coefficients of the stage's
// point.  Returns the magnitude of the terms summed into the derivatives
// (eta_I + k_I |I|): the scale of their FP32 rounding noise.
//
// FtPoint: what the Faraday-thick mode needs of a stage point besides the
// coefficients, 1 / |lambda|^2 and max(|k_Q|, |k_C|) / |lambda| (lambda = k_I -
// i k_F): it does not depend on the state either.
struct FtPoint {
  float il, cpl;
};
__device__ __forceinline__ FtPoint ft_point(const Coef32& c) {
  const float il = 1.f / fmaf(c.kI, c.kI, c.kF * c.kF);
  return FtPoint{il, fmaxf(fabsf(c.kQ), fabsf(c.kC)) * sqrtf(il)};
}

template <bool FULL>
__device__ __forceinline__ float stokes_rhs(const Coef32& c, const FtPoint& q, const float* y, float cs, float sn,
                                            float* dk, bool ft, float* cpl) {
  const float scale = fabsf(c.eI) + fabsf(c.kI * y[0]);
  if (!FULL) {
    dk[0] = c.eI - c.kI * y[0];
    return scale;
  }
  if (kFtm) {
    // Faraday-thick mode: the lab-frame polarisation Pi = Q + iU obeys
    // Pi' = -lambda Pi + S, lambda = k_I - i k_F, S = (eta_Q - k_Q I) - i k_C V.
    // Where |lambda| is far above the rate at which S / lambda changes, Pi is
    // that quasi-static value plus a transient d whose rotating-frame value
    // only decays (d' = -k_I d, up to the adiabatic lag); I and V see the
    // quasi-static part through k_Q Re Pi and k_C Im Pi, the transient's
    // share rotates at k_F and integrates to at most ~cpl |d|.  dk[1], dk[2]
    // carry the rotating-frame value e^{-i chi} S / lambda itself.  Both modes
    // are formed and selected: a warp mostly has lanes in each, and its six
    // stages stay free of branches (with the points' FtPoint formed together:
    // 3.57 G evaluations 56.0 -> 52.6 ms, 24.5 M on groups 5.50 -> 5.06).
    const float sQ = c.eQ - c.kQ * y[0], sU = -c.kC * y[3];
    const float pre = fmaf(sQ, c.kI, -sU * c.kF) * q.il, pim = fmaf(sQ, c.kF, sU * c.kI) * q.il;
    const float Ql = ft ? pre : cs * y[1] - sn * y[2], Ul = ft ? pim : sn * y[1] + cs * y[2];
    dk[0] = c.eI - c.kI * y[0] - c.kQ * Ql - c.kV * y[3];
    dk[1] = ft ? fmaf(cs, pre, sn * pim) : -c.kI * y[1] + cs * sQ + sn * sU;
    dk[2] = ft ? fmaf(-sn, pre, cs * pim) : -c.kI * y[2] - sn * sQ + cs * sU;
    dk[3] = c.eV - c.kI * y[3] - c.kV * y[0] + c.kC * Ul;
    dk[4] = c.kF;
    if (ft) *cpl = q.cpl;
    return scale;
  }
  float Qlab = cs * y[1] - sn * y[2];
  float Ulab = sn * y[1] + cs * y[2];
  float sQ = c.eQ - c.kQ * y[0];
  float sU = -c.kC * y[3];
  dk[0] = c.eI - c.kI * y[0] - c.kQ * Qlab - c.kV * y[3];
  dk[1] = -c.kI * y[1] + cs * sQ + sn * sU;
  dk[2] = -c.kI * y[2] - sn * sQ + cs * sU;
  dk[3] = c.eV - c.kI * y[3] - c.kV * y[0] + c.kC * Ulab;
  dk[4] = c.kF;
  return scale;
}

// Local equilibrium of the transfer equation dx/dt = eps - K x at the IQUV
// start point of an optically thick ray (the end of the tau step that landed
// on tau_eq): x = K^-1 eps with the lab-frame transfer matrix of the
// reference's full-Stokes system (src/System.cpp:41-63; k_U = eta_U = h_Q = 0
// in its frame)
//     K = [[k_I, k_Q, 0, k_V], [k_Q, k_I, k_F, 0], [0, -k_F, k_I, k_C],
//          [k_V, 0, -k_C, k_I]],  eps = (eta_I, eta_Q, 0, eta_V),
// solved in FP64 by Gaussian elimination (K's symmetric part is positive
// definite: |k_Q|, |k_V| < k_I).  chi = 0 there, so the rotating frame is the
// lab frame.  The state is in the request's scaled intensity units, like the
// coefficients.  (ox, oy, oz): the start point [cm].
template <bool GENERAL>
__device__ __noinline__ float4 equilibrium_state(const JshRequest* __restrict__ reqs, int r, int f, double ox,
                                                double oy, double oz) {
  const JshRequest& R = reqs[r];
  Coef32 c;
  coef32_rt<GENERAL>(R, R.mix, R.mix.fc[f], f3((float)(ox * INV_PC), (float)(oy * INV_PC), (float)(oz * INV_PC)), COEF_FULL, c);
  double A[4][5] = {{c.kI, c.kQ, 0.0, c.kV, c.eI},
                    {c.kQ, c.kI, c.kF, 0.0, c.eQ},
                    {0.0, -c.kF, c.kI, c.kC, 0.0},
                    {c.kV, 0.0, -c.kC, c.kI, c.eV}};
  // no pivoting: every leading block of K has a positive definite symmetric
  // part, so its pivots are nonzero
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!(A[k][k] != 0.0)) return make_float4(0.f, 0.f, 0.f, 0.f);  // k_I = 0 there: zero state
#pragma unroll
    for (int i = k + 1; i < 4; ++i) {
      const double m = A[i][k] / A[k][k];
#pragma unroll
      for (int j = k; j < 5; ++j) A[i][j] -= m * A[k][j];
    }
  }
  double x[4];
#pragma unroll
  for (int i = 3; i >= 0; --i) {
    double a = A[i][4];
#pragma unroll
    for (int j = i + 1; j < 4; ++j) a -= A[i][j] * x[j];
    x[i] = a / A[i][i];
  }
  return make_float4((float)x[0], (float)x[1], (float)x[2], (float)x[3]);
}

__device__ __forceinline__ void lane_finish_iquv(Lane& L, const JshRequest* __restrict__ reqs, Tally& T, bool lead) {
  L.phase = PH_IDLE;
  if (!lead) return;
  write_finished_iquv(reqs, L.r, L.f, L.h, L.chi.hi, L.chi.lo, L.x[0], L.x[1], L.x[2], L.x[3], L.status, L.evals0,
                      L.evals);
  tally_add(T, reqs, L.r, L.evals, L.acc, L.rej, L.status);
}

// First item slot of part `part`'s emitted items in iq_items / iq_order.
__device__ __forceinline__ uint32_t iq_first(const JshRequest& R, int part) {
  return part ? R.buckets[JSH_RANK_DEEP] * (uint32_t)R.n_nu : 0u;
}

// Split form, IQUV kernel: start work item w (heaviest-first over the
// batch's emitted items) where the tau kernel left it -- the I/IQUV pass's
// first segment, start point and state (zero, or the local equilibrium).
template <bool GENERAL>
__device__ __forceinline__ void lane_start_iquv(Lane& L, const JshRequest* __restrict__ reqs,
                                                const unsigned long long* base, int n_req, unsigned long long w,
                                                int part) {
  const int r = find_request(base, n_req, w);
  const JshRequest& R = reqs[r];
  const JshIquvItem it = R.iq_items[R.iq_order[iq_first(R, part) + (uint32_t)(w - base[r])]];
  L.r = r;
  L.f = it.f;
  L.h = it.h;
  L.phase = PH_IQUV;
  L.nseg = (int8_t)(it.flags & 3);
  L.first_seg = (int8_t)((it.flags >> 3) & 3) - 1;
  const bool eq = (it.flags & 4) != 0;
  L.first_div = it.first_div;
  L.t_first = it.t_first;
  L.chi = DF{0.f, 0.f};
  L.x[0] = L.x[1] = L.x[2] = L.x[3] = 0.f;
  L.status = it.status;
  L.evals0 = it.evals;
  L.evals = L.acc = L.rej = 0;
  L.tri = -1;
  L.ft = 0;
  L.ft_cool = 0;
  L.seg = L.first_seg >= 0 ? L.first_seg : L.nseg - 1;
  const JshHit& H = R.hits[L.h];
  if (eq) {
    const int s = L.seg;
    const double tc = L.t_first * JSH_PC;
    const float4 xe = equilibrium_state<GENERAL>(reqs, L.r, L.f, H.seg[s][0] + R.plane.rx * tc, H.seg[s][1] + R.plane.ry * tc,
                                        H.seg[s][2] + R.plane.rz * tc);
    L.x[0] = xe.x;
    L.x[1] = xe.y;
    L.x[2] = xe.z;
    L.x[3] = xe.w;
  }
  begin_iquv_segment<PASS_IQUV>(L, R);
}

// FP32 unit roundoff; the Stokes error norm's noise floor is
// kNoise * h * scale.  The rounding noise of the embedded error estimate of
// a Stokes component is about 0.3 u h scale (four terms of magnitude
// <= scale per derivative, weighted by |e_j| <= 0.05).
constexpr float kNoise = 5.9604645e-8f;
// Faraday-thick mode of the IQUV pass: entry where
// |k_F| >= kFtRatio k_I; the quasi-static part's lag and the transient's
// left-out coupling must stay within kFtTol (atol + rtol I); after a refused
// entry or an exit the mode waits kFtCooldown accepted steps, after an entry
// estimate that found the transient too large kFtRetry, doubled for each
// such estimate in a row (up to 255).
constexpr float kFtRatio = 100.f;
constexpr float kFtTol = 1.f;
constexpr uint8_t kFtCooldown = 32;
constexpr int kFtRetry = 16;  // accepted steps after an entry estimate that found the transient too large
constexpr float kFtAxis = 0.25f;  // largest step / distance from the jet axis
// The mode's tolerance scales with I, as the full mode's own control of
// (Q, U) does through its noise floor (the quasi-static |Q + iU| is ~k_I/k_F
// of I where the mode applies).
__device__ __forceinline__ float ft_tolerance(float I, float rtol, float atol) {
  return kFtTol * fmaf(rtol, fabsf(I), atol);
}

// ---------------------------------------------------------------- tau pass
// The tau pass integrates dtau/dt = k_I along each segment.  Its right-hand
// side does not depend on the state, so the pass is a quadrature: each step
// is a Gauss-Kronrod 7/15 panel (jsh_quadrature.h) of adaptive width, with
// the adaptive-range semantics of the reference's Dormand-Prince pass
// (src/Observation.cpp:150-211: steps end exactly at the segment's end,
// dt_max bounds them, tau_max is located by bisection) and its tolerances
// (tau_atol, tau_rtol of the running segment depth).  A panel of 15 k_I
// evaluations replaces a step of 6: on the conical jet a tau pass needs
// ~2.3x fewer evaluations (an FP64 experiment on 600 C1 items: 75-97 per
// item against 195, errors 1e-9 .. 1e-12 of the converged depth).
__constant__ float c_gk_t[15] = {
    (float)(0.5 * (1.0 + jsh_gk15_x[0])),  (float)(0.5 * (1.0 + jsh_gk15_x[1])),
    (float)(0.5 * (1.0 + jsh_gk15_x[2])),  (float)(0.5 * (1.0 + jsh_gk15_x[3])),
    (float)(0.5 * (1.0 + jsh_gk15_x[4])),  (float)(0.5 * (1.0 + jsh_gk15_x[5])),
    (float)(0.5 * (1.0 + jsh_gk15_x[6])),  (float)(0.5 * (1.0 + jsh_gk15_x[7])),
    (float)(0.5 * (1.0 + jsh_gk15_x[8])),  (float)(0.5 * (1.0 + jsh_gk15_x[9])),
    (float)(0.5 * (1.0 + jsh_gk15_x[10])), (float)(0.5 * (1.0 + jsh_gk15_x[11])),
    (float)(0.5 * (1.0 + jsh_gk15_x[12])), (float)(0.5 * (1.0 + jsh_gk15_x[13])),
    (float)(0.5 * (1.0 + jsh_gk15_x[14]))};
__constant__ float c_gk_wk[15] = {
    (float)(0.5 * jsh_gk15_wk[0]),  (float)(0.5 * jsh_gk15_wk[1]),  (float)(0.5 * jsh_gk15_wk[2]),
    (float)(0.5 * jsh_gk15_wk[3]),  (float)(0.5 * jsh_gk15_wk[4]),  (float)(0.5 * jsh_gk15_wk[5]),
    (float)(0.5 * jsh_gk15_wk[6]),  (float)(0.5 * jsh_gk15_wk[7]),  (float)(0.5 * jsh_gk15_wk[8]),
    (float)(0.5 * jsh_gk15_wk[9]),  (float)(0.5 * jsh_gk15_wk[10]), (float)(0.5 * jsh_gk15_wk[11]),
    (float)(0.5 * jsh_gk15_wk[12]), (float)(0.5 * jsh_gk15_wk[13]), (float)(0.5 * jsh_gk15_wk[14])};
__constant__ float c_gk_wg[15] = {
    (float)(0.5 * jsh_gk15_wg[0]),  (float)(0.5 * jsh_gk15_wg[1]),  (float)(0.5 * jsh_gk15_wg[2]),
    (float)(0.5 * jsh_gk15_wg[3]),  (float)(0.5 * jsh_gk15_wg[4]),  (float)(0.5 * jsh_gk15_wg[5]),
    (float)(0.5 * jsh_gk15_wg[6]),  (float)(0.5 * jsh_gk15_wg[7]),  (float)(0.5 * jsh_gk15_wg[8]),
    (float)(0.5 * jsh_gk15_wg[9]),  (float)(0.5 * jsh_gk15_wg[10]), (float)(0.5 * jsh_gk15_wg[11]),
    (float)(0.5 * jsh_gk15_wg[12]), (float)(0.5 * jsh_gk15_wg[13]), (float)(0.5 * jsh_gk15_wg[14])};
__constant__ float c_gk_wd[15] = {
    (float)(0.5 * (jsh_gk15_wk[0] - jsh_gk15_wg[0])),   (float)(0.5 * (jsh_gk15_wg[1] - jsh_gk15_wk[1])),
    (float)(0.5 * (jsh_gk15_wk[2] - jsh_gk15_wg[2])),   (float)(0.5 * (jsh_gk15_wg[3] - jsh_gk15_wk[3])),
    (float)(0.5 * (jsh_gk15_wk[4] - jsh_gk15_wg[4])),   (float)(0.5 * (jsh_gk15_wg[5] - jsh_gk15_wk[5])),
    (float)(0.5 * (jsh_gk15_wk[6] - jsh_gk15_wg[6])),   (float)(0.5 * (jsh_gk15_wg[7] - jsh_gk15_wk[7])),
    (float)(0.5 * (jsh_gk15_wk[8] - jsh_gk15_wg[8])),   (float)(0.5 * (jsh_gk15_wg[9] - jsh_gk15_wk[9])),
    (float)(0.5 * (jsh_gk15_wk[10] - jsh_gk15_wg[10])), (float)(0.5 * (jsh_gk15_wg[11] - jsh_gk15_wk[11])),
    (float)(0.5 * (jsh_gk15_wk[12] - jsh_gk15_wg[12])), (float)(0.5 * (jsh_gk15_wg[13] - jsh_gk15_wk[13])),
    (float)(0.5 * (jsh_gk15_wk[14] - jsh_gk15_wg[14]))};
// Floor of a panel's tolerance on its error estimate K - G = h sum (w_K -
// w_G)_i k_i: each FP32 k_i carries a relative rounding error of up to
// ~2.6e-6 (exp2 of arguments up to ~60 in the log-domain coefficient form),
// so |K - G| is never resolved below 2.6e-6 h sum |w_K - w_G|_i |k_i|.  The
// floor is ~10x that: |K - G| bounds the Gauss rule's error, the Kronrod
// value kept is far more accurate, and panel widths grow only as the 15th
// root of the tolerance (on the 512x1024 conical jet 3x the noise bound and
// this floor gave 130 and 124 evaluations per tau pass, both with the
// worst tau 1.7e-6 off the converged oracle).
constexpr float kPanelNoise = 3e-5f;
// Bisection limit of the tau_max crossing inside a panel.
constexpr int kCrossIters = 48;

// The end of an item's tau pass: finish it (tau <= tau_min), hand it to the
// IQUV kernel (PASS_TAU) or start its I/IQUV pass in the same lane.
template <int PASS, bool GENERAL>
__device__ __forceinline__ void tau_pass_done(Lane& L, const JshRequest* __restrict__ reqs, const JshMixed& X,
                                              int part, Tally& T, bool lead) {
  const JshRequest& R = reqs[L.r];
  // a depth of one segment surely above tau_min stays a pair (no FP64 here)
  const bool pair = PASS == PASS_TAU && L.seg == 0 && L.tau_seg.hi > X.tau_min_f;
  if (!pair) {
    L.tau_bg = tau_total(L);
    if (!(L.tau_bg > R.P.tau_min)) {
      lane_finish(L, reqs, T, lead);
      return;
    }
  }
  L.status |= JSH_ST_IQUV;
  L.phase = PH_IQUV;
  bool eq = false;
  if (L.first_seg >= 0 && X.eq_start) {
    // the equilibrium start needs depth behind tau_eq: rays shallower than
    // eq_min are integrated whole from their far end
    if ((pair ? df_val(L.tau_seg) : L.tau_bg) >= X.eq_min || (L.status & JSH_ST_TAU_CROSSED)) eq = true;
    else L.first_seg = -1;
  }
  if (PASS == PASS_TAU) {
    L.phase = PH_IDLE;
    if (!lead) return;
    emit_iquv(reqs, part, L.r, L.f, L.h, pair, L.tau_seg, L.tau_bg, L.thick, L.t_first, L.first_seg, L.nseg, eq,
              L.status, L.evals);
    tally_add(T, reqs, L.r, L.evals, L.acc, L.rej, 0u);
    return;
  }
  L.first_div = first_step_divisor(L.tau_bg, R.P.n);
  L.seg = L.first_seg >= 0 ? L.first_seg : L.nseg - 1;
  L.tri = -1;  // as the IQUV kernel's fresh lanes
  L.ft = 0;
  L.ft_cool = 0;
  const JshHit& H = R.hits[L.h];
  if (eq) {
    const int s = L.seg;
    const double tc = L.t_first * JSH_PC;
    const float4 xe = equilibrium_state<GENERAL>(reqs, L.r, L.f, H.seg[s][0] + R.plane.rx * tc, H.seg[s][1] + R.plane.ry * tc,
                                        H.seg[s][2] + R.plane.rz * tc);
    L.x[0] = xe.x;
    L.x[1] = xe.y;
    L.x[2] = xe.z;
    L.x[3] = xe.w;
  }
  begin_iquv_segment<PASS>(L, R);
}

// One panel of an active lane's tau pass (or a segment / pass transition).
// While the lane bisects a tau_max crossing (L.init set; the tau pass has
// no other use for it), the panel [t, t + w] with w the midpoint of the
// bracket [k1[0], k1[1]] is evaluated instead.
template <int PASS, bool GENERAL, int NG>
__device__ __forceinline__ void tau_panel_step(Lane& L, const JshRequest* __restrict__ reqs, const JshMixed& X,
                                               float* Ksh, int part, Tally& T, const LaneGroup& grp) {
  const JshRequest& R = reqs[L.r];
  const JshFreqConst F = X.fc[L.f];
  const bool bis = L.init;
  // integration direction: +d (away from the observer)
  const F3 dir = f3(-X.nl[0], -X.nl[1], -X.nl[2]);
  bool at_bp = false;
  if (!bis) {
    const DF rem = df_sub(L.length, L.t);
    const float remf = rem.hi + rem.lo;
    if (!(remf > 0.f)) goto segment_done;
    if (X.dt_max_f != 0.f && L.dt > X.dt_max_f) L.dt = X.dt_max_f;
    if (L.k1[2] < INFINITY) {
      // the segment's closest approach to the jet axis lies ahead: panels
      // close in on it by factors of 4 down to the approach distance and
      // end on it
      const DF rb = df_sub(DF{L.k1[2], 0.f}, L.t);
      const float rbf = rb.hi + rb.lo;
      if (rbf > 0.f) {
        L.dt = fminf(L.dt, fmaxf(0.75f * rbf, L.k1[3]));
        if (!(L.dt < rbf)) {
          L.dt = rbf;
          at_bp = true;
        }
      } else {
        L.k1[2] = INFINITY;
      }
    }
    L.last = !(L.dt < remf);
    if (L.last) {
      L.dt = remf;
      at_bp = false;
    }
  }
  if (L.nsteps++ >= R.P.max_steps) {
    L.status |= JSH_ST_STEP_LIMIT;
    goto abort;
  }
  {
    const float h = bis ? 0.5f * (L.k1[0] + L.k1[1]) : L.dt;
    const F3 pn = f3(L.bx, L.by, L.bz);
    float K = 0.f, G = 0.f, A = 0.f;
    if (NG == 1) {
#pragma unroll 1
      for (int i = 0; i < 15; ++i) {
        Coef32 c;
        coef32_rt<GENERAL>(R, X, F, pn + dir * (c_gk_t[i] * h), COEF_KI, c, L.h, (uint32_t)L.f, L.evals + (uint32_t)i);
        K = fmaf(c_gk_wk[i], c.kI, K);
        G = fmaf(c_gk_wg[i], c.kI, G);
        A = fmaf(c_gk_wd[i], fabsf(c.kI), A);
      }
    } else if (NG > 1) {
      // three nodes a lane, then the sums in the nodes' order
      float k3[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        Coef32 c;
        coef32_rt<GENERAL>(R, X, F, pn + dir * (c_gk_t[kGroupLanes * j + grp.sub] * h), COEF_KI, c);
        k3[j] = c.kI;
      }
#pragma unroll
      for (int i = 0; i < 15; ++i) {
        const float kI = __shfl_sync(grp.mask, k3[i / kGroupLanes], grp.base + i % kGroupLanes);
        K = fmaf(c_gk_wk[i], kI, K);
        G = fmaf(c_gk_wg[i], kI, G);
        A = fmaf(c_gk_wd[i], fabsf(kI), A);
      }
    } else {
      grp.sync();  // the panel before has read its nodes
#pragma unroll 1
      for (int i = grp.sub; i < 15; i += grp.n) {
        Coef32 c;
        coef32_rt<GENERAL>(R, X, F, pn + dir * (c_gk_t[i] * h), COEF_KI, c);
        Ksh[i] = c.kI;
      }
      grp.sync();
#pragma unroll 1
      for (int i = 0; i < 15; ++i) {
        const float kI = Ksh[i];
        K = fmaf(c_gk_wk[i], kI, K);
        G = fmaf(c_gk_wg[i], kI, G);
        A = fmaf(c_gk_wd[i], fabsf(kI), A);
      }
    }
    L.evals += 15;
    K *= h;
    G *= h;
    if (!(K == K) || isinf(K)) {
      L.status |= JSH_ST_NAN;
      goto abort;
    }
    if (bis) {
      // tau at t + h against tau_max; stop within tau_precision of it
      // (src/Observation.cpp:166-185).  The crossing point starts the
      // I/IQUV pass; tau keeps the crossing panel's end value, as the
      // reference keeps the crossing step's (src/Observation.cpp:208).
      L.rej++;
      const double dv = df_val(df_add(L.tau_seg, K)) - R.P.tau_max;
      const bool done = fabs(dv) <= R.P.tau_precision || !(L.k1[1] - L.k1[0] > 1e-7f * L.k1[1]);
      if (!done && ++L.fails < kCrossIters) {
        if (dv > 0.0) L.k1[1] = h;
        else L.k1[0] = h;
        return;
      }
      if (!done) L.status |= JSH_ST_BISECT_LIMIT;
      L.init = false;
      L.tau_seg = DF{L.k1[2], L.k1[3]};
      L.first_seg = L.seg;
      L.t_first = df_val(L.t) + (double)h;
      L.nseg = L.seg + 1;
      tau_pass_done<PASS, GENERAL>(L, reqs, X, part, T, (grp.sub == 0));
      return;
    }
    // error test: |K - G| against the tolerance of the running depth, never
    // below the FP32 noise floor of the estimate
    const float err = fabsf(K - G);
    const float tol = fmaf(X.tau_rtol, fabsf(L.tau_seg.hi) + fabsf(K), X.tau_atol) + kPanelNoise * h * A;
    const float r = err > 0.f ? tol / err : 1e30f;
    if (!(r >= 1.f)) {
      L.dt = h * fminf(fmaxf(0.9f * __powf(r, 1.0f / 15.0f), 0.2f), 0.9f);
      L.last = false;
      L.rej++;
      if (++L.fails >= dp::FAIL_LIMIT) {
        L.status |= JSH_ST_FAIL_LIMIT;
        goto abort;
      }
      return;
    }
    // landing on the optically thick depth: a panel may not overshoot
    // tau_thick by more than 25 %, so that the IQUV pass can start at the end
    // of the crossing panel, where tau is as accurate as the integration
    if (L.first_seg < 0 && L.tau_seg.hi < L.thick_left && L.tau_seg.hi + K > 1.25f * L.thick_left) {
      L.dt = h * fmaxf((1.1f * L.thick_left - L.tau_seg.hi) / K, 0.01f);
      L.last = false;
      L.rej++;
      if (++L.fails >= dp::FAIL_LIMIT) {
        L.status |= JSH_ST_FAIL_LIMIT;
        goto abort;
      }
      return;
    }
    // tau_max inside this panel (the pass ends here): a crossing panel may
    // not overshoot tau_max by more than 25 % either (tau keeps its end
    // value); when no optically thick start precedes the crossing, the I/IQUV
    // pass starts at the crossing point, bisected for inside the panel
    {
      const DF tn = df_add(L.tau_seg, K);
      if (tn.hi > X.tau_max_hi || (tn.hi == X.tau_max_hi && tn.lo >= X.tau_max_lo)) {
        if (tn.hi > 1.25f * X.tau_max_hi) {
          L.dt = h * fmaxf((1.1f * X.tau_max_hi - L.tau_seg.hi) / K, 0.01f);
          L.last = false;
          L.rej++;
          if (++L.fails >= dp::FAIL_LIMIT) {
            L.status |= JSH_ST_FAIL_LIMIT;
            goto abort;
          }
          return;
        }
        L.status |= JSH_ST_TAU_CROSSED;
        L.acc++;
        if (L.first_seg < 0) {
          L.init = true;
          L.k1[0] = 0.f;
          L.k1[1] = h;
          L.k1[2] = tn.hi;
          L.k1[3] = tn.lo;
          L.fails = 0;
          return;
        }
        L.tau_seg = tn;
        L.nseg = L.seg + 1;
        tau_pass_done<PASS, GENERAL>(L, reqs, X, part, T, (grp.sub == 0));
        return;
      }
    }
    // accept
    const DF t_prev = L.t;
    const DF t_new = L.last ? L.length : df_add(L.t, h);
    if (t_new.hi == t_prev.hi && t_new.lo == t_prev.lo) {
      L.status |= JSH_ST_DT_UNDERFLOW;
      goto abort;
    }
    L.t = t_new;
    L.bx = df_axpy_round(t_new, DF{X.dhi[0], X.dlo[0]}, L.p0x);
    L.by = df_axpy_round(t_new, DF{X.dhi[1], X.dlo[1]}, L.p0y);
    L.bz = df_axpy_round(t_new, DF{X.dhi[2], X.dlo[2]}, L.p0z);
    L.fails = 0;
    L.acc++;
    L.dt = h * fminf(fmaxf(0.9f * __powf(fminf(r, 1e15f), 1.0f / 15.0f), 1.f), 4.f);
    if (at_bp) {
      // past the closest approach: start again at the approach distance
      L.k1[2] = INFINITY;
      L.dt = L.k1[3];
    }
    L.tau_seg = df_add(L.tau_seg, K);
    if (L.first_seg < 0 && L.tau_seg.hi >= L.thick_left) {
      // optically thick from here on (tau within [1, 1.25] tau_thick): the
      // IQUV pass starts at the end of this panel; the tau pass goes on for
      // the tau image
      L.first_seg = L.seg;
      L.t_first = df_val(t_new);
    }
    return;
  }

segment_done : {
  if (L.seg + 1 < L.nseg) {
    L.seg++;
    begin_tau_segment<PASS>(L, R, X);
    return;
  }
  tau_pass_done<PASS, GENERAL>(L, reqs, X, part, T, (grp.sub == 0));
  return;
}

abort:
  L.init = false;
  L.tau_bg = tau_total(L);
  lane_finish(L, reqs, T, (grp.sub == 0));
}

// One Dormand-Prince attempt of an active lane's tau pass (the reference's
// stepper, src/Observation.cpp:150-211), for the requests whose fields may
// jump (sheaths, composite laws, cells, random and gridded fields: a
// quadrature panel's error estimate can miss a jump between its nodes).
// dtau/dt = k_I does not depend on the state, so only the last stage
// combination (the increment) is formed.
template <int PASS, bool GENERAL>
__device__ __forceinline__ void tau_dopri_step(Lane& L, const JshRequest* __restrict__ reqs, const JshMixed& X,
                                               float* K, int part, Tally& T, const LaneGroup& grp) {
  const JshRequest& R = reqs[L.r];
  const JshFreqConst F = X.fc[L.f];
  const F3 dirf = f3(-X.nl[0], -X.nl[1], -X.nl[2]);
  const float max_dt = X.dt_max_f;
  const float atol = X.tau_atol;
  const float rtol = X.tau_rtol;
  {
    const DF rem = df_sub(L.length, L.t);
    const float remf = rem.hi + rem.lo;
    if (!(remf > 0.f)) goto segment_done;
    L.last = !(L.dt < remf);
    if (L.last) L.dt = remf;
  }
  if (L.nsteps++ >= R.P.max_steps) {
    L.status |= JSH_ST_STEP_LIMIT;
    goto abort;
  }
  if (max_dt != 0.f && fabsf(L.dt) > max_dt) {
    L.dt = max_dt;
    L.rej++;
    if (++L.fails >= dp::FAIL_LIMIT) {
      L.status |= JSH_ST_FAIL_LIMIT;
      goto abort;
    }
    return;
  }
  {
    const F3 pn = f3(L.bx, L.by, L.bz);
    const float h = L.dt;
    if (!L.init) {
      Coef32 c;
      coef32_rt<GENERAL>(R, X, F, pn, COEF_KI, c, L.h, (uint32_t)L.f, L.evals, &L.tri);
      L.k1[0] = c.kI;
      L.evals++;
      L.init = true;
    }
    // k_I does not depend on the state, and the last two stages share their
    // point (c = 1): five evaluations serve the six stages, unless every
    // evaluation draws its own random direction
    grp.sync();  // the step before has read its stages
    if (grp.sub == 0) K[0] = L.k1[0];
    const int np = R.model.rnd_kind == JSH_RND_POINTS ? 6 : 5;
#pragma unroll 1
    for (int s = grp.sub + 1; s <= np; s += grp.n) {
      Coef32 c;
      // the sixth point is the group's first lane's alone
      coef32_rt<GENERAL>(R, X, F, pn + dirf * (c_C[s] * h), COEF_KI, c, L.h, (uint32_t)L.f,
                         L.evals + (uint32_t)(s - 1), &L.tri, s <= 5 ? grp : single_lane());
      K[s] = c.kI;
      if (s == 5 && np == 5) K[6] = c.kI;
    }
    grp.sync();
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 6; ++j) acc = fmaf(dp_a32(6, j), K[j], acc);
    const float inc = h * acc;
    L.evals += 6;
    float a = 0.f;
#pragma unroll
    for (int j = 0; j < 7; ++j) a = fmaf(c_E[j], K[j], a);
    const float adt = fabsf(h);
    // no cancellation in dtau/dt = k_I: the plain odeint norm
    const float e = fabsf(h * a) / fmaf(rtol, fmaf(adt, fabsf(L.k1[0]), fabsf(L.tau_seg.hi)), atol);
    if (!(e == e) || isinf(e)) {
      L.status |= JSH_ST_NAN;
      goto abort;
    }
    if (e > 1.0f) {
      const float f = 0.9f * __powf(e, -1.0f / 3.0f);
      L.dt = h * (f > 0.2f ? f : 0.2f);
      if (max_dt != 0.f && fabsf(L.dt) > max_dt) L.dt = max_dt;
      L.rej++;
      if (++L.fails >= dp::FAIL_LIMIT) {
        L.status |= JSH_ST_FAIL_LIMIT;
        goto abort;
      }
      return;
    }
    // landing on the optically thick depth (as the panels)
    if (L.first_seg < 0 && L.tau_seg.hi < L.thick_left && L.tau_seg.hi + inc > 1.25f * L.thick_left) {
      L.dt = h * fmaxf((1.1f * L.thick_left - L.tau_seg.hi) / inc, 0.01f);
      L.last = false;
      L.rej++;
      if (++L.fails >= dp::FAIL_LIMIT) {
        L.status |= JSH_ST_FAIL_LIMIT;
        goto abort;
      }
      return;
    }
    const DF t_prev = L.t;
    const DF t_new = L.last ? L.length : df_add(L.t, h);
    if (t_new.hi == t_prev.hi && t_new.lo == t_prev.lo) {
      L.status |= JSH_ST_DT_UNDERFLOW;
      goto abort;
    }
    L.t = t_new;
    L.bx = df_axpy_round(t_new, DF{X.dhi[0], X.dlo[0]}, L.p0x);
    L.by = df_axpy_round(t_new, DF{X.dhi[1], X.dlo[1]}, L.p0y);
    L.bz = df_axpy_round(t_new, DF{X.dhi[2], X.dlo[2]}, L.p0z);
    L.fails = 0;
    L.acc++;
    if (e < 0.5f) {
      const float ee = e > 0.00032f ? e : 0.00032f;
      L.dt = h * (0.9f * __powf(ee, -0.2f));
      if (max_dt != 0.f && fabsf(L.dt) > max_dt) L.dt = max_dt;
    }
    const DF tau_prev = L.tau_seg;
    L.tau_seg = df_add(L.tau_seg, inc);
    if (L.first_seg < 0 && L.tau_seg.hi >= L.thick_left) {
      L.first_seg = L.seg;
      L.t_first = df_val(t_new);
    }
    if (L.tau_seg.hi > X.tau_max_hi || (L.tau_seg.hi == X.tau_max_hi && L.tau_seg.lo >= X.tau_max_lo)) {
      L.status |= JSH_ST_TAU_CROSSED;
      const double t_old = df_val(t_prev);
      double tc = crossing_time(df_val(tau_prev), t_old, (double)h, h, K[0], K[2], K[3], K[4], K[5], K[6], inc,
                                R.P.tau_max, R.P.tau_precision);
      if (tc < 0.0) {
        // the reference keeps bisecting; stop at the last bracket's midpoint
        L.status |= JSH_ST_BISECT_LIMIT;
        tc = t_old + 0.5 * (double)h;
      }
      if (L.first_seg < 0 || (L.first_seg == L.seg && tc < L.t_first)) {
        L.first_seg = L.seg;
        L.t_first = tc;
      }
      L.nseg = L.seg + 1;
      tau_pass_done<PASS, GENERAL>(L, reqs, X, part, T, (grp.sub == 0));
      return;
    }
    L.k1[0] = K[6];
    return;
  }

segment_done : {
  if (L.seg + 1 < L.nseg) {
    L.seg++;
    begin_tau_segment<PASS>(L, R, X);
    return;
  }
  tau_pass_done<PASS, GENERAL>(L, reqs, X, part, T, (grp.sub == 0));
  return;
}

abort:
  L.tau_bg = tau_total(L);
  lane_finish(L, reqs, T, (grp.sub == 0));
}

// One step of an active lane's tau pass: a quadrature panel for the smooth
// benchmark family (helical conical B and BK n in the plasma frame, flat
// flow), a Dormand-Prince attempt otherwise.  The choice belongs to the
// request, so every build of the kernels gives the same bits.
template <int PASS, bool GENERAL, int NG>
__device__ __forceinline__ void tau_step(Lane& L, const JshRequest* __restrict__ reqs, const JshMixed& X, float* K,
                                         int part, Tally& T, const LaneGroup& grp) {
  if (!GENERAL || X.helical_log) tau_panel_step<PASS, GENERAL, NG>(L, reqs, X, K, part, T, grp);
  else tau_dopri_step<PASS, GENERAL>(L, reqs, X, K, part, T, grp);
}

// A stage point's coefficients in shared memory: words, or two float4 (NG > 1).
template <bool FULL, int NG>
__device__ __forceinline__ void put_coefficients(float* q, const Coef32& c) {
  if (NG >= 1 && FULL) {
    reinterpret_cast<float4*>(q)[0] = make_float4(c.kI, c.eI, c.kQ, c.kV);
    reinterpret_cast<float4*>(q)[1] = make_float4(c.kF, c.kC, c.eQ, c.eV);
    return;
  }
  q[0] = c.kI;
  q[1] = c.eI;
  if (FULL) {
    q[2] = c.kQ;
    q[3] = c.kV;
    q[4] = c.kF;
    q[5] = c.kC;
    q[6] = c.eQ;
    q[7] = c.eV;
  }
}
template <bool FULL, int NG>
__device__ __forceinline__ void get_coefficients(const float* q, Coef32& c) {
  if (NG >= 1 && FULL) {
    const float4 a = reinterpret_cast<const float4*>(q)[0], b = reinterpret_cast<const float4*>(q)[1];
    c = Coef32{a.x, a.z, a.w, b.x, b.y, a.y, b.z, b.w};
    return;
  }
  c.kI = q[0];
  c.eI = q[1];
  if (FULL) {
    c.kQ = q[2];
    c.kV = q[3];
    c.kF = q[4];
    c.kC = q[5];
    c.eQ = q[6];
    c.eV = q[7];
  }
}

// ------------------------------------------------------- I / IQUV pass
// One Dormand-Prince attempt (or a segment transition) of an active lane in
// its I/IQUV pass, towards the observer.  The arithmetic is the same in
// every form (static, single-kernel, split), so the images are bitwise the
// same.
template <bool FULL, int PASS, bool GENERAL, int NG>
__device__ __forceinline__ void lane_step(Lane& L, const JshRequest* __restrict__ reqs, const JshMixed& X, float* Q,
                                          Tally& T, const LaneGroup& grp) {
  constexpr int NK = StageWidth<FULL>::NK;
  constexpr int NX = StageWidth<FULL>::NX;
  const JshRequest& R = reqs[L.r];
  const JshFreqConst F = X.fc[L.f];
  const F3 dirf = f3(X.nl[0], X.nl[1], X.nl[2]);
  // error-norm tolerances in FP32 (the norm needs a few digits; t and dt stay FP64)
  const float atol = F.atol;
  const float rtol = X.rtol;

  if (kFtm && FULL && L.ft) {
    // Faraday-thick mode: its steps follow I and V only, so nothing else
    // keeps them from straddling the narrow features of the field where a
    // ray passes the jet axis (the dip of B_perp, the reversal of the
    // azimuthal field within the approach distance): a step spans at most
    // kFtAxis of the point's distance from the axis.  Where that is under a
    // radian of rotation the full integration is as fast: leave the mode.
    const float cap = kFtAxis * sqrtf(fmaf(L.bx, L.bx, L.by * L.by));
    if (cap * fabsf(L.k1[NK - 1]) < 1.f) {
      L.ft = 0;
      L.ft_cool = kFtCooldown;
      L.init = false;
      L.dt = fminf(L.dt, 1.f / fabsf(L.k1[NK - 1]));
    } else {
      L.dt = fminf(L.dt, cap);
    }
  }
  // integrate_adaptive / adaptive range: finish at exactly t = length (a
  // step that would pass the end is shortened to end there)
  {
    const DF rem = df_sub(L.length, L.t);
    const float remf = rem.hi + rem.lo;
    if (!(remf > 0.f)) goto segment_done;
    L.last = !(L.dt < remf);
    if (L.last) L.dt = remf;
  }
  if (L.nsteps++ >= R.P.max_steps) {
    L.status |= JSH_ST_STEP_LIMIT;
    goto abort;
  }
  {
    const F3 pn = f3(L.bx, L.by, L.bz);
    // frame rotation at the step start: FP32 sincos of the (reduced) angle
    float c0 = 1.f, s0 = 0.f;
    if (FULL) sincosf(L.chi.hi, &s0, &c0);
    const float h = L.dt;
    const bool ft = kFtm && FULL && L.ft;
    float cpl = 0.f;  // Faraday-thick mode: max(|k_Q|, |k_C|) / |lambda| of the last evaluation
    constexpr int mode = FULL ? COEF_FULL : COEF_I;
    // first derivative from the coefficients at the step's start; false: the
    // Faraday-thick mode was refused there
    auto first = [&](const Coef32& c) {
      L.s1 = stokes_rhs<FULL>(c, ft ? ft_point(c) : FtPoint{}, L.x, c0, s0, L.k1, ft, &cpl);
      L.kI1 = c.kI;
      L.evals++;
      L.init = true;
      if (ft) {
        // entry: the transient carried in, d = (q, u) - e^{-i chi} S / lambda,
        // must be small enough that the rotating coupling the mode leaves
        // out of I and V stays within the tolerance
        const float dq = L.x[1] - L.k1[1], du = L.x[2] - L.k1[2];
        if (!(cpl * sqrtf(fmaf(dq, dq, du * du)) <= ft_tolerance(L.x[0], rtol, atol))) {
          L.ft = 0;
          L.ft_cool = kFtCooldown;
          L.init = false;
          return false;
        }
      }
      return true;
    };
    constexpr bool kLoop = NG == 1 && FULL;  // the start's evaluation is in the points' loop
    if (!kLoop && !L.init) {
      Coef32 c;
      coef32_rt<GENERAL>(R, X, F, pn, mode, c, L.h, (uint32_t)L.f, L.evals0 + L.evals, &L.tri);
      if (!first(c)) return;
    }
    // The coefficients depend on the stage's point alone, not on the state,
    // and the last two stages share their point (c = 1): all five points are
    // evaluated before the stages, so that their chains of dependent
    // operations overlap.  The fused build of Stokes I keeps them in registers;
    // the others in shared memory, with one copy of the coefficients' code, and
    // a sixth point where every evaluation draws a random direction.
    Coef32 C[5];
    FtPoint P[5] = {};
    // words of a point (a fused group's: two float4, three with the
    // Faraday-thick mode)
    constexpr int kPoint = NG > 1 ? (kFtm ? 12 : 8) : StageWidth<FULL>::NC;
    const bool six = GENERAL && R.model.rnd_kind == JSH_RND_POINTS;
    if (kLoop) {
      // one copy of the coefficients' code (six copies were more than the
      // instruction caches hold: the warps waited for instructions a third of
      // the time) and 128 registers instead of 149: 517 550 items 897 -> 850 us,
      // 705 176 1.39 -> 1.37 ms, Faraday-thick 3.57 G evaluations 55.6 -> 51.2 ms.
      // Stokes I alone is faster unrolled (530 against 590 us).
      bool in_mode = true;
#pragma unroll 1
      for (int s = L.init ? 1 : 0; s <= 5; ++s) {
        Coef32 c;
        coef32_rt<GENERAL>(R, X, F, pn + dirf * (c_C[s] * h), mode, c);
        if (s == 0) in_mode = first(c);
        else put_coefficients<FULL, NG>(Q + (s - 1) * kPoint, c);
      }
      if (!in_mode) return;
      if (ft) {
#pragma unroll
        for (int s = 0; s < 5; ++s) {
          Coef32 c;
          get_coefficients<FULL, NG>(Q + s * kPoint, c);
          P[s] = ft_point(c);
        }
      }
    } else if (NG == 1) {
#pragma unroll
      for (int s = 1; s <= 5; ++s)
        coef32_rt<GENERAL>(R, X, F, pn + dirf * (dp_c32(s) * h), mode, C[s - 1]);
    } else {
      grp.sync();  // the step before has read its coefficients
      const int np = six ? 6 : 5;
#pragma unroll 1
      for (int s = grp.sub + 1; s <= (NG > 1 ? 5 : np); s += NG > 1 ? NG : grp.n) {
        Coef32 c;
        // a sixth point is the group's first lane's alone
        coef32_rt<GENERAL>(R, X, F, pn + dirf * (c_C[s] * h), mode, c, L.h, (uint32_t)L.f,
                           L.evals0 + L.evals + (uint32_t)(s - 1), &L.tri, s <= 5 ? grp : single_lane());
        put_coefficients<FULL, NG>(Q + (s - 1) * kPoint, c);
        if (NG > 1 && kFtm && FULL && ft) {
          const FtPoint q = ft_point(c);
          Q[(s - 1) * kPoint + 8] = q.il;
          Q[(s - 1) * kPoint + 9] = q.cpl;
        }
      }
      grp.sync();
    }
    float K[7][NK];
#pragma unroll
    for (int c = 0; c < NK; ++c) K[0][c] = L.k1[c];
    float inc[NK];
    float smax = L.s1, s7 = 0.f, kI7 = 0.f;
    auto stage = [&](auto S) {
      constexpr int s = decltype(S)::value;
      float acc[NK];
      combine_stage<s, NK>(K, acc);
      float y[4], dk[5];
#pragma unroll
      for (int c = 0; c < 4; ++c) y[c] = (c < NX) ? fmaf(h, acc[c < NK ? c : 0], L.x[c]) : 0.f;
      float cs = c0, sn = s0;
      if (FULL) {
        float sd, cd;
        __sincosf(h * acc[NK - 1], &sd, &cd);
        cs = c0 * cd - s0 * sd;
        sn = s0 * cd + c0 * sd;
      }
      Coef32 c;
      const float* q = Q + (s == 6 ? (six ? 5 : 4) : s - 1) * kPoint;
      if (NG != 1 || kLoop) get_coefficients<FULL, NG>(q, c);
      else c = C[s == 6 ? 4 : s - 1];
      FtPoint cq{};
      if (NG == 1) cq = P[s == 6 ? 4 : s - 1];
      else if (ft && NG > 1) cq = FtPoint{q[8], q[9]};
      else if (ft) cq = ft_point(c);
      const float sc = stokes_rhs<FULL>(c, cq, y, cs, sn, dk, ft, &cpl);
      smax = fmaxf(smax, sc);
      s7 = sc;
      kI7 = c.kI;
      if (ft && s < 6) {
        // Faraday-thick mode: the inner stages' (q, u) slots are free (no
        // stage point uses (q, u)); they keep the stage's k_I and its coupling
        // factor, or +inf where rotation does not outrun absorption a
        // hundredfold (a reversal of the line-of-sight field inside the step,
        // as on rays past the axis of a helical field, breaks the
        // quasi-static picture between the step's ends)
        dk[2] = fabsf(dk[NK - 1]) >= kFtRatio * kI7 ? cpl : INFINITY;
        dk[1] = kI7;
      }
#pragma unroll
      for (int c = 0; c < NK; ++c) K[s][c] = dk[c];
      if (s == 6) {
#pragma unroll
        for (int c = 0; c < NK; ++c) inc[c] = h * acc[c];
      }
    };
    stage(std::integral_constant<int, 1>());
    stage(std::integral_constant<int, 2>());
    stage(std::integral_constant<int, 3>());
    stage(std::integral_constant<int, 4>());
    stage(std::integral_constant<int, 5>());
    stage(std::integral_constant<int, 6>());
    L.evals += 6;
    // embedded error estimate and odeint's default error checker:
    // max_i |err_i| / (atol + rtol (|x_i| + |dt| |x'_i|))
    float err[NK];
#pragma unroll
    for (int c = 0; c < NK; ++c) {
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < 7; ++j) a = fmaf(dp_e32(j), K[j][c], a);
      err[c] = h * a;
    }
    // FP32 resolution floor: an error estimate below the rounding noise of
    // the terms it is computed from carries no information, so the
    // tolerance never drops below kNoise * h * (their magnitude)
    const float adt = fabsf(h);
    const float floor_ = kNoise * adt * smax;
    float e = 0.f;
    {
      // q', u', V in an optically thick step (optical depth h k_I > 0.01):
      // their source terms are small differences of terms of size ~scale
      // (e_Q - k_Q I, ...) and the rounding noise of their error estimate
      // reaches ~0.7 of the floor, which pins the estimate in odeint's
      // no-growth band [0.5, 1] (95 % of the core rays' steps were there).
      // A 100x floor there (an allowed error of 6e-6 h scale per step, damped
      // by the optical depth in front) took the 512x1024 conical jet's
      // longest item from 4 585 to 2 689 evaluations (10x: 34 % fewer than
      // 1x); against the converged oracle V rose from 3.4e-7 to 1.7e-6 of
      // max I, I and Q stayed.  Optically thin steps keep the 1x floor
      // (their Q/U control is what keeps far rays from stepping over the
      // narrow dip of B_perp where they pass the jet axis).
      const float fl_pol = (adt * fabsf(L.kI1) > 0.01f) ? 100.f * floor_ : floor_;
#pragma unroll
      for (int c = 0; c < NX; ++c) {
        if (ft && (c == 1 || c == 2)) continue;  // (Q, U) is not integrated in the Faraday-thick mode
        const float fl = (c == 0) ? floor_ : fl_pol;
        float r = fabsf(err[c]) / (fmaf(rtol, fmaf(adt, fabsf(L.k1[c]), fabsf(L.x[c])), atol) + fl);
        e = fmaxf(e, r);
      }
      if (ft) {
        // adiabatic condition of the quasi-static part: its lag behind
        // S / lambda, (d/dt (S / lambda)) / lambda, estimated over the step
        // from the lab-frame values at its ends, and the transient's left-out
        // coupling stay within the tolerance; else the step is redone in the
        // full mode (from the same state: (q, u) is the full polarisation in
        // both modes)
        float cs6, sn6;  // the frame at the step's end, as its last stage had it
        {
          float sd, cd;
          __sincosf(inc[NK - 1], &sd, &cd);
          cs6 = c0 * cd - s0 * sd;
          sn6 = s0 * cd + c0 * sd;
        }
        float cpl_max = cpl;
        bool ft_ok = fabsf(K[6][NK - 1]) >= kFtRatio * kI7;
#pragma unroll
        for (int j = 1; j < 6; ++j) cpl_max = fmaxf(cpl_max, K[j][2]);
        ft_ok = ft_ok && cpl_max < INFINITY;
        const float ft_tol = ft_tolerance(L.x[0], rtol, atol);
        const float p0r = c0 * K[0][1] - s0 * K[0][2], p0i = s0 * K[0][1] + c0 * K[0][2];
        const float p6r = cs6 * K[6][1] - sn6 * K[6][2], p6i = sn6 * K[6][1] + cs6 * K[6][2];
        const float dr = p6r - p0r, di = p6i - p0i;
        const float lam = sqrtf(fmaf(kI7, kI7, K[6][NK - 1] * K[6][NK - 1]));
        const float dq = L.x[1] - K[0][1], du = L.x[2] - K[0][2];
        if (!ft_ok || !(sqrtf(fmaf(dr, dr, di * di)) <= adt * lam * ft_tol) ||
            !(cpl_max * sqrtf(fmaf(dq, dq, du * du)) <= ft_tol)) {
          L.ft = 0;
          L.ft_cool = kFtCooldown;
          L.init = false;
          L.dt = fminf(h, 1.f / fabsf(L.k1[NK - 1]));
          return;
        }
      }
      if (FULL && !ft) {
        // a rotation error d chi moves (Q, U) by P d chi; the lab-frame norm
        // of the reference would compare that with rtol (P + h |dQ/dt|),
        // and |dQ/dt| ~ k_F P there
        float P = sqrtf(fmaf(L.x[1], L.x[1], L.x[2] * L.x[2]));
        e = fmaxf(e, fabsf(err[NK - 1]) * P / (fmaf(rtol * P, fmaf(adt, fabsf(L.k1[NK - 1]), 1.f), atol) + floor_));
      }
    }
    if (!(e == e) || isinf(e)) {
      L.status |= JSH_ST_NAN;
      goto abort;
    }
    if (e > 1.0f) {
      float f = 0.9f * __powf(e, -1.0f / 3.0f);
      L.dt = h * (f > 0.2f ? f : 0.2f);
      L.rej++;
      if (++L.fails >= dp::FAIL_LIMIT) {
        L.status |= JSH_ST_FAIL_LIMIT;
        goto abort;
      }
      return;
    }
    // accept
    const DF t_prev = L.t;
    const DF t_new = L.last ? L.length : df_add(L.t, h);
    if (t_new.hi == t_prev.hi && t_new.lo == t_prev.lo) {
      L.status |= JSH_ST_DT_UNDERFLOW;
      goto abort;
    }
    L.t = t_new;
    L.bx = df_axpy_round(t_new, DF{-X.dhi[0], -X.dlo[0]}, L.p0x);
    L.by = df_axpy_round(t_new, DF{-X.dhi[1], -X.dlo[1]}, L.p0y);
    L.bz = df_axpy_round(t_new, DF{-X.dhi[2], -X.dlo[2]}, L.p0z);
    L.fails = 0;
    L.acc++;
    if (e < 0.5f) {
      float ee = e > 0.00032f ? e : 0.00032f;
      L.dt = h * (0.9f * __powf(ee, -0.2f));
    }
    float qn = 0.f, un = 0.f;
    if (ft) {
      // quasi-static part at the end plus the transient, decayed by the
      // step's optical depth (h sum b_j k_I,j over the stages)
      float btau = dp_a32(6, 0) * L.kI1;
#pragma unroll
      for (int j = 1; j < 6; ++j) btau = fmaf(dp_a32(6, j), K[j][1], btau);
      const float decay = expf(-h * btau);
      qn = fmaf(L.x[1] - K[0][1], decay, K[6][1]);
      un = fmaf(L.x[2] - K[0][2], decay, K[6][2]);
    }
#pragma unroll
    for (int c = 0; c < NX; ++c) L.x[c] += inc[c];
    if (ft) {
      L.x[1] = qn;
      L.x[2] = un;
    }
    if (FULL) {
      L.chi = df_add(L.chi, inc[NK - 1]);
      if (fabsf(L.chi.hi) > 3.14159265f) {
        // subtract k 2 pi exactly: 2 pi = c_hi + c_lo, k c_hi = p + pe
        const float k = rintf(L.chi.hi * 0.159154943f);
        const float c_hi = 6.28318548f, c_lo = -1.74845553e-7f;
        const float pr = k * c_hi, pe = fmaf(k, c_hi, -pr);
        L.chi = df_add(df_add(L.chi, -pr), -fmaf(k, c_lo, pe));
      }
    }
#pragma unroll
    for (int c = 0; c < NK; ++c) L.k1[c] = K[6][c];
    L.s1 = s7;
    L.kI1 = kI7;
    if (kFtm && FULL && !ft) {
      // rotation outruns absorption a hundredfold and turns (q, u) by a
      // noticeable angle per step: try the Faraday-thick mode, whose steps
      // follow I and V, if the transient it would carry looks small enough.
      // The estimate needs no evaluation: this step's last one gives the
      // rotating-frame source e^{-i chi} S = (q, u)' + k_I (q, u), so the
      // quasi-static value and the transient d = (q, u) - e^{-i chi} S / lambda
      // follow, and |d| k_I / |lambda| stands in for the left-out coupling
      // (k_Q, k_C < k_I for synchrotron gas; the first evaluation in the mode
      // checks the entry with the coefficients themselves).
      const float kF = L.k1[NK - 1];
      if (L.ft_cool) L.ft_cool--;
      else if (fabsf(kF) >= kFtRatio * kI7 && fabsf(kF) * h >= 0.01f) {
        const float sr = fmaf(kI7, L.x[1], L.k1[1]), si = fmaf(kI7, L.x[2], L.k1[2]);
        const float il = __fdividef(1.f, fmaf(kI7, kI7, kF * kF));  // an estimate: the fast reciprocal will do
        const float dq = L.x[1] - fmaf(sr, kI7, -si * kF) * il, du = L.x[2] - fmaf(sr, kF, si * kI7) * il;
        const float tol = ft_tolerance(L.x[0], rtol, atol);
        if (kI7 * kI7 * il * fmaf(dq, dq, du * du) <= tol * tol) {
          L.ft = 1;
          L.init = false;
          L.ft_back = 0;
        } else {
          // back off: 16, 32, 64, 128, then 255 steps between estimates
          L.ft_cool = (uint8_t)min(255, kFtRetry << L.ft_back);
          if (L.ft_back < 4) L.ft_back++;
        }
      }
    }
    if (!L.last) return;
  }

segment_done : {
  if (L.seg > 0) {
    L.seg--;
    begin_iquv_segment<PASS>(L, R);
    return;
  }
  if (PASS == PASS_IQUV) {
    lane_finish_iquv(L, reqs, T, (grp.sub == 0));
    return;
  }
  lane_finish(L, reqs, T, (grp.sub == 0));
  return;
}

abort:
  if (PASS == PASS_IQUV) {
    lane_finish_iquv(L, reqs, T, (grp.sub == 0));
    return;
  }
  lane_finish(L, reqs, T, (grp.sub == 0));
}

// One step of an active lane in whichever pass it is (one lane per item).
template <bool FULL, int PASS>
__device__ __forceinline__ void lane_advance(Lane& L, const JshRequest* __restrict__ reqs, float* Q, Tally& T) {
  const LaneGroup one = single_lane();
  const JshMixed& X = reqs[L.r].mix;
  if (PASS == PASS_BOTH && L.phase == PH_TAU) tau_step<PASS, true, 0>(L, reqs, X, Q, 0, T, one);
  else lane_step<FULL, PASS, true, 0>(L, reqs, X, Q, T, one);
}

// A persistent warp's work: every idle lane (or group of lanes) takes the next
// item of the queue once at least `refill` lanes of the warp idle (with groups
// the two that belong to none among them), `start(w)`
// begins item w on this lane, `step()` advances an active one.  Returns once
// the queue is empty and at most `leave` of the warp's items are unfinished.
//
// `deal`: the warps begin without the queue, the k-th lane or group of every
// warp with the k-th stretch of the order, so that the longest items are in
// different warps.  `drained`: there is nothing left to begin.
template <typename Start, typename Step>
__device__ __forceinline__ void run_queue(Lane& L, unsigned long long* queue, unsigned long long total, int refill,
                                          const LaneGroup& grp, bool deal, bool drained, int leave, Start start,
                                          Step step) {
  const bool member = grp.mask != 0;
  const unsigned before = (1u << (grp.base & 31)) - 1u;
  const int slots = grp.n == 1 ? 32 : kWarpGroups;
  unsigned long long dealt = 0;
  if (deal) {
    const unsigned warps = gridDim.x * (blockDim.x / 32), warp = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const unsigned long long w = (unsigned long long)(grp.base / grp.n) * warps + warp;
    if (member && w < total) start(w);
    dealt = (unsigned long long)slots * warps;
  }
  bool exhausted = drained;
  for (;;) {
    const unsigned idle = __ballot_sync(0xffffffffu, member && L.phase == PH_IDLE && grp.sub == 0);
    const int nidle = __popc(idle);
    if (!exhausted && (32 - (slots - nidle) * grp.n >= refill || nidle == slots) && nidle > 0) {
      unsigned long long b = 0;
      if ((threadIdx.x & 31u) == 0) b = atomicAdd(queue, (unsigned long long)nidle);
      b = __shfl_sync(0xffffffffu, b, 0);
      b += dealt;
      if (b + (unsigned long long)nidle >= total) exhausted = true;
      if (member && L.phase == PH_IDLE) {
        const unsigned long long w = b + (unsigned long long)__popc(idle & before);
        if (w < total) start(w);
      }
    }
    const unsigned active = __ballot_sync(0xffffffffu, L.phase != PH_IDLE);
    if (exhausted && (active == 0 || __popc(active) <= leave)) break;
    if (L.phase != PH_IDLE) step();
  }
}

// Hand the warp's unfinished items of single lanes (kWarpGroups at most) to
// its groups: the k-th to the k-th group, whose lanes then hold its state.
// An item in its I/IQUV pass only, on a field that is not gridded.
__device__ __forceinline__ void spread_items(Lane& L, const LaneGroup& grp) {
  __syncwarp();  // the lanes have read their stage storage
  const unsigned active = __ballot_sync(0xffffffffu, L.phase != PH_IDLE);
  const int k = grp.base / kGroupLanes;
  const bool has = grp.mask != 0 && k < __popc(active);
  const int src = has ? (int)__fns(active, 0, k + 1) : 0;
  auto from = [&](auto& v) { v = __shfl_sync(0xffffffffu, v, src); };
  auto from_df = [&](DF& v) { from(v.hi), from(v.lo); };
  auto from_byte = [&](auto& v) {
    int i = (int)v;
    from(i);
    v = (std::remove_reference_t<decltype(v)>)i;
  };
  from(L.r), from(L.f), from(L.h);
  from_byte(L.phase), from_byte(L.seg), from_byte(L.first_seg), from_byte(L.init);
  from_byte(L.ft), from_byte(L.ft_cool), from_byte(L.ft_back);
  from_df(L.p0x), from_df(L.p0y), from_df(L.p0z);
  from(L.bx), from(L.by), from(L.bz);
  from_df(L.length), from_df(L.t);
  from(L.dt), from(L.first_div), from(L.t_first);
  from_df(L.chi);
#pragma unroll
  for (int c = 0; c < 4; ++c) from(L.x[c]);
#pragma unroll
  for (int c = 0; c < 5; ++c) from(L.k1[c]);
  from(L.s1), from(L.kI1);
  from(L.nsteps), from(L.fails), from(L.status);
  from(L.evals), from(L.acc), from(L.rej), from(L.evals0);
  if (!has) L.phase = PH_IDLE;
}

// Place of this lane's group among the CTA's groups (the last one for a lane
// that belongs to none).
__device__ __forceinline__ int group_slot(const LaneGroup& grp) {
  return (int)(threadIdx.x / 32) * kWarpGroups + min(grp.base / kGroupLanes, kWarpGroups - 1);
}

// Whether a launch of `total` items runs them on groups of lanes: up to
// `slots_factor` items for each group the grid holds.
__device__ __forceinline__ bool on_groups(unsigned long long total, int slots_factor) {
  return total <= (unsigned long long)slots_factor * gridDim.x * (blockDim.x / 32) * kWarpGroups;
}

// Words of stage storage of a lane that runs both passes.
template <bool FULL>
__device__ __host__ constexpr int form_words() {
  return StageWidth<FULL>::kWords > kTauWords ? StageWidth<FULL>::kWords : kTauWords;
}

// Dynamic shared memory of a CTA: the lanes' stage storage (`lanes` false, the
// fused IQUV build: kLaneWords of them, none for Stokes I), or that of its groups.
template <bool FULL>
constexpr size_t stage_smem(int block, bool lanes = true) {
  const size_t one = sizeof(float) * (size_t)block * (lanes ? form_words<FULL>() : FULL ? kLaneWords : 0);
  const size_t groups = sizeof(float) * kGroupWords * kWarpGroups * (size_t)(block / 32);
  return one > groups ? one : groups;
}

}  // namespace

}  // namespace jsh
