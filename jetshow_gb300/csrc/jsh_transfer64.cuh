// jsh_transfer64.cuh -- the all-FP64 per-(ray, frequency) transfer on the
// device: tau pass front to back with the dense-output Dormand-Prince
// stepper stopping at tau_max (src/Observation.cpp:126-214), then the I or
// IQUV pass back to front with the controlled stepper of
// integrate_adaptive (src/Observation.cpp:242-308; the IQUV right-hand side
// of src/System.cpp:41-63).
//
// Dormand-Prince 5(4) tableau: Dormand & Prince (1980).  Dense output:
// Hairer, Norsett & Wanner, Solving ODEs I, II.6.  Step control as
// documented for Boost.Odeint's controlled_runge_kutta / default_error_checker
// (error = max_i |e_i| / (atol + rtol (|x_i| + |dt| |x'_i|)), decrease
// max(0.9 err^-1/3, 0.2), increase 0.9 max(err, 5^-5)^-1/5 when err < 0.5,
// 500 consecutive rejections abort) and integrate_adaptive's truncation of
// the last step to the interval end.
#pragma once

#include <float.h>

#include "jsh_fields.cuh"
#include "jsh_request.h"

namespace jsh {

namespace dp {
constexpr double C2 = 1.0 / 5, C3 = 3.0 / 10, C4 = 4.0 / 5, C5 = 8.0 / 9;
constexpr double A21 = 1.0 / 5;
constexpr double A31 = 3.0 / 40, A32 = 9.0 / 40;
constexpr double A41 = 44.0 / 45, A42 = -56.0 / 15, A43 = 32.0 / 9;
constexpr double A51 = 19372.0 / 6561, A52 = -25360.0 / 2187, A53 = 64448.0 / 6561, A54 = -212.0 / 729;
constexpr double A61 = 9017.0 / 3168, A62 = -355.0 / 33, A63 = 46732.0 / 5247, A64 = 49.0 / 176,
                 A65 = -5103.0 / 18656;
constexpr double B1 = 35.0 / 384, B3 = 500.0 / 1113, B4 = 125.0 / 192, B5 = -2187.0 / 6784, B6 = 11.0 / 84;
constexpr double E1 = 71.0 / 57600, E3 = -71.0 / 16695, E4 = 71.0 / 1920, E5 = -17253.0 / 339200,
                 E6 = 22.0 / 525, E7 = -1.0 / 40;
constexpr double D1 = -12715105075.0 / 11282082432.0, D3 = 87487479700.0 / 32700410799.0,
                 D4 = -10690763975.0 / 1880347072.0, D5 = 701980252875.0 / 199316789632.0,
                 D6 = -1453857185.0 / 822651844.0, D7 = 69997945.0 / 29380423.0;
constexpr int FAIL_LIMIT = 500;
}  // namespace dp

// Tableau rows of stages 2..7 (row 7 = the 5th-order weights b).
__device__ __forceinline__ constexpr double dp_a(int s, int j) {
  switch (s * 8 + j) {
    case 8: return dp::A21;
    case 16: return dp::A31;
    case 17: return dp::A32;
    case 24: return dp::A41;
    case 25: return dp::A42;
    case 26: return dp::A43;
    case 32: return dp::A51;
    case 33: return dp::A52;
    case 34: return dp::A53;
    case 35: return dp::A54;
    case 40: return dp::A61;
    case 41: return dp::A62;
    case 42: return dp::A63;
    case 43: return dp::A64;
    case 44: return dp::A65;
    case 48: return dp::B1;
    case 50: return dp::B3;
    case 51: return dp::B4;
    case 52: return dp::B5;
    case 53: return dp::B6;
    default: return 0.0;
  }
}
// Path point(t) = p0 + t * dir; nl = LOS towards the observer.
struct Path64 {
  D3 p0, dir, nl;
  Freq64 F;
  Frame64 flat;       // kinematics of a constant flat flow
  uint32_t rk0, rk1;  // random-direction key of the item: pixel, frequency
  // coefficients at path coordinate t for the item's evaluation `ev`
  template <int MODE>
  __device__ __forceinline__ void at(const JshModel& m, double t, double* k, uint32_t ev) const {
    coefficients64<MODE>(m, F, flat, p0 + dir * t, nl, k, rk0, rk1, ev);
  }
};
__device__ __forceinline__ Path64 path64(const JshModel& m, D3 p0, D3 dir, D3 nl, double nu, uint32_t rk0 = 0,
                                         uint32_t rk1 = 0) {
  Path64 P{p0, dir, nl, freq64(m, nu), Frame64{}, rk0, rk1};
  if (m.v_kind == JSH_V_CONST_FLAT) P.flat = frame64(m, p0, nl);
  return P;
}

struct Ctl64 {
  double atol, rtol, max_dt;
  int64_t max_steps;
  uint64_t acc, rej, evals;
};

// ------------------------------------------------------------ lane groups
// An item runs on a group of five lanes of one warp (six groups a warp, the
// last two lanes idle).  The coefficients of a Dormand-Prince step depend on
// the stage's point alone, not on the state, and its last two stages share
// their point (c = 1): lane k evaluates the point of stage k + 2 and the five
// results are exchanged, so a step costs one evaluation's instructions
// instead of six.  GB300 holds a sub-partition's FP64 pipe ~64 cycles for a
// warp instruction, however many lanes take part, so an item's time is its
// number of FP64 instructions, and five lanes an item serve large images too:
// against a lane per item, 64x96 pixels of the conical jet 64.3 -> 4.8 ms (a
// fifth of the sub-partitions was busy), 256x384 233 -> 50 ms, Stokes I of a
// tangled field at 512x768 50 -> 47 ms, 64x64 of a gridded jet 21.3 -> 1.03 s.
// The step control is carried by every lane alike (the same values, so the
// same branches); of the IQUV state each lane advances one component.
constexpr int kGroup = 5;
constexpr int kGroupsPerWarp = 6;

struct Group64 {
  unsigned mask;   // the group's lanes
  int base, sub;   // its first lane, this lane's place in it
  double* sh;      // FULL: the step's coefficients [5][NCOEF] (this group's)
};

__device__ __forceinline__ Group64 group_of(double* sh_warp) {
  const int lane = (int)(threadIdx.x & 31u);
  const int g = lane / kGroup;
  return Group64{g < kGroupsPerWarp ? 0x1fu << (kGroup * g) : 0u, kGroup * g, lane - kGroup * g,
                 sh_warp + (g < kGroupsPerWarp ? g : 0) * kGroup * NCOEF};
}
__device__ __forceinline__ double from_lane(const Group64& G, double v, int k) {
  return __shfl_sync(G.mask, v, G.base + k);
}

// One new step size for a rejected or an accepted step (one pow).
__device__ __forceinline__ double next_dt(double dt, double e, bool rejected, double max_dt) {
  if (!rejected && !(e < 0.5)) return dt;
  const double lo = 0.00032;  // 5^-5
  const double f = 0.9 * pow(rejected || e > lo ? e : lo, rejected ? -1.0 / 3.0 : -1.0 / 5.0);
  dt *= rejected ? (f > 0.2 ? f : 0.2) : f;
  if (max_dt != 0.0 && fabs(dt) > max_dt) dt = max_dt;
  return dt;
}

// steps_schedule (src/utils.cpp:354-366) with its default tau limits.
__device__ __forceinline__ int steps_schedule(double tau, int n_min, int n_max) {
  const double tau_min = 0.1, tau_max = 100.0;
  if (tau <= tau_min) return n_min;
  if (tau >= tau_max) return n_max;
  double b = -log(tau_min);
  double k = n_max / pow((log(tau_max) + b), 2.0);
  double n = k * pow((log(tau) + b), 2.0) + n_min;
  return (int)ceil(n);
}

struct ItemOut {
  double tau, l, iquv[4];
  uint32_t status;
};

// The coefficients at point t + c dt of this lane's stage (lane k: stage
// k + 2), keyed as the (k + 1)-th of the step's evaluations.
template <int MODE>
__device__ __forceinline__ void stage_coefficients(const JshModel& m, const Path64& P, const Group64& G, double t,
                                                   double dt, uint32_t ev, double* k) {
  const double c = G.sub == 0 ? dp::C2 : G.sub == 1 ? dp::C3 : G.sub == 2 ? dp::C4 : G.sub == 3 ? dp::C5 : 1.0;
  P.at<MODE>(m, t + c * dt, k, ev + (uint32_t)G.sub);
}

// Tau pass of one segment (src/Observation.cpp:150-211): dense-output
// Dormand-Prince steps of dtau/dt = k_I over [0, length] until tau_max.
// Returns a failure status or 0; x the depth, x_old / t_old / dt_used / k the
// last accepted step for the dense output.
__device__ __forceinline__ uint32_t tau_segment64(const JshModel& m, const Path64& P, const Group64& G, Ctl64& C,
                                                  double length, double dt, double tau_max, uint32_t& ev, double& x,
                                                  double& x_old, double& t_old, double& dt_used, double (&k)[7],
                                                  bool& crossed) {
  double t = 0.0;
  int64_t nsteps = 0;
  int fails = 0;
  {
    double c[NCOEF];
    if (!(length - t > DBL_EPSILON)) return 0;
    P.at<0>(m, 0.0, c, ev++);
    C.evals++;
    k[0] = c[CK_I];
  }
  for (;;) {  // one attempt
    if (fails == 0) {
      if (!(length - t > DBL_EPSILON)) return 0;
      if ((t + dt) - length > DBL_EPSILON) dt = length - t;
    }
    if (nsteps++ >= C.max_steps) return JSH_ST_STEP_LIMIT;
    if (C.max_dt != 0.0 && fabs(dt) > C.max_dt) {
      dt = C.max_dt;
      C.rej++;
      if (++fails >= dp::FAIL_LIMIT) return JSH_ST_FAIL_LIMIT;
      continue;
    }
    double c[NCOEF];
    stage_coefficients<0>(m, P, G, t, dt, ev, c);
#pragma unroll
    for (int s = 1; s < 6; ++s) k[s] = from_lane(G, c[CK_I], s - 1);
    k[6] = k[5];
    if (m.rnd_kind == JSH_RND_POINTS) {  // every evaluation draws its own direction: a sixth one
      P.at<0>(m, t + dt, c, ev + 5);
      k[6] = c[CK_I];
    }
    ev += 6;
    C.evals += 6;
    double acc = dp_a(6, 0) * k[0];
#pragma unroll
    for (int j = 1; j < 6; ++j) acc += dp_a(6, j) * k[j];
    const double xn = x + dt * acc;
    const double err = dt * (dp::E1 * k[0] + dp::E3 * k[2] + dp::E4 * k[3] + dp::E5 * k[4] + dp::E6 * k[5] +
                             dp::E7 * k[6]);
    const double e = fabs(err) / (C.atol + C.rtol * (fabs(x) + fabs(dt) * fabs(k[0])));
    if (isnan(e)) return JSH_ST_NAN;
    const bool rejected = e > 1.0;
    const double t_new = t + dt;
    if (!rejected && t_new == t) return JSH_ST_DT_UNDERFLOW;
    const double used = dt;
    dt = next_dt(dt, e, rejected, C.max_dt);
    if (rejected) {
      C.rej++;
      if (++fails >= dp::FAIL_LIMIT) return JSH_ST_FAIL_LIMIT;
      continue;
    }
    fails = 0;
    C.acc++;
    x_old = x;
    x = xn;
    t_old = t;
    dt_used = used;
    t = t_new;
    if (x >= tau_max) {
      crossed = true;
      return 0;
    }
    k[0] = k[6];
  }
}

// I / IQUV pass of one segment (src/Observation.cpp:242-308): controlled
// steps of dx/dt over [0, length].  FULL: lane k < 4 of the group carries
// component k of (I, Q, U, V) in x (lane 4 repeats lane 3), whose derivative
// (src/System.cpp:41-63) is A - k_I x - B x_p - C x_q with
//   I: A = eta_I, (B, p) = (k_Q, Q), (C, q) = (k_V, V)
//   Q: A = eta_Q, (k_Q, I), (k_F, U)        U: A = 0, (-k_F, Q), (k_C, V)
//   V: A = eta_V, (k_V, I), (-k_C, U);
// otherwise every lane carries I.
template <bool FULL>
__device__ __forceinline__ uint32_t iquv_segment64(const JshModel& m, const Path64& P, const Group64& G, Ctl64& C,
                                                   double length, double dt, uint32_t& ev, double& x) {
  const int comp = FULL ? (G.sub < 3 ? G.sub : 3) : 0;
  const int ia = comp == 0 ? CE_I : comp == 1 ? CE_Q : CE_V;
  const int ib = comp < 2 ? CK_Q : comp == 2 ? CK_F : CK_V, ip = comp == 0 || comp == 2 ? 1 : 0;
  const int ic = comp == 0 ? CK_V : comp == 1 ? CK_F : CK_C, iq = comp == 0 || comp == 2 ? 3 : 2;
  // derivative of the lane's component at the state whose component is y
  auto rhs = [&](const double* c, double y) {
    if (!FULL) return c[CE_I] - c[CK_I] * y;
    const double yp = from_lane(G, y, ip), yq = from_lane(G, y, iq);
    const double a = comp == 2 ? 0.0 : c[ia], b = comp == 2 ? -c[ib] : c[ib], d = comp == 3 ? -c[ic] : c[ic];
    return a - c[CK_I] * y - b * yp - d * yq;
  };
  double t = 0.0, k[7];
  int64_t nsteps = 0;
  int fails = 0;
  {
    if (!(length - t > DBL_EPSILON)) return 0;
    double c[NCOEF];
    P.at<FULL ? 2 : 1>(m, 0.0, c, ev++);
    C.evals++;
    if (FULL) {
      __syncwarp(G.mask);
      if (G.sub == 0)
#pragma unroll
        for (int i = 0; i < NCOEF; ++i) G.sh[i] = c[i];
      __syncwarp(G.mask);
      k[0] = rhs(G.sh, x);
    } else {
      k[0] = rhs(c, x);
    }
  }
  for (;;) {  // one attempt
    if (fails == 0) {
      if (!(length - t > DBL_EPSILON)) return 0;
      if ((t + dt) - length > DBL_EPSILON) dt = length - t;
    }
    if (nsteps++ >= C.max_steps) return JSH_ST_STEP_LIMIT;
    double c[NCOEF], c6[NCOEF];
    stage_coefficients<FULL ? 2 : 1>(m, P, G, t, dt, ev, c);
    const bool six = m.rnd_kind == JSH_RND_POINTS;
    if (six) P.at<FULL ? 2 : 1>(m, t + dt, c6, ev + 5);
    ev += 6;
    C.evals += 6;
    if (FULL) {
      __syncwarp(G.mask);  // the step before has read its coefficients
#pragma unroll
      for (int i = 0; i < NCOEF; ++i) G.sh[G.sub * NCOEF + i] = c[i];
      __syncwarp(G.mask);
    }
    double y = x;
#pragma unroll
    for (int s = 1; s < 7; ++s) {
      double acc = dp_a(s, 0) * k[0];
#pragma unroll
      for (int j = 1; j < s; ++j) acc += dp_a(s, j) * k[j];
      y = x + dt * acc;
      if (FULL) {
        if (s == 6 && six) {
          __syncwarp(G.mask);
          if (G.sub == 4)
#pragma unroll
            for (int i = 0; i < NCOEF; ++i) G.sh[4 * NCOEF + i] = c6[i];
          __syncwarp(G.mask);
        }
        k[s] = rhs(G.sh + (s < 6 ? s - 1 : 4) * NCOEF, y);
      } else {
        double ci[2];
        ci[CK_I] = from_lane(G, c[CK_I], s < 6 ? s - 1 : 4);
        double ei = from_lane(G, c[CE_I], s < 6 ? s - 1 : 4);
        if (s == 6 && six) {
          ci[CK_I] = c6[CK_I];
          ei = c6[CE_I];
        }
        k[s] = ei - ci[CK_I] * y;
      }
    }
    const double err = dt * (dp::E1 * k[0] + dp::E3 * k[2] + dp::E4 * k[3] + dp::E5 * k[4] + dp::E6 * k[5] +
                             dp::E7 * k[6]);
    const double r = fabs(err) / (C.atol + C.rtol * (fabs(x) + fabs(dt) * fabs(k[0])));
    double e = r;
    bool bad = isnan(r);
    if (FULL) {
      e = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double ri = from_lane(G, r, i);
        bad |= isnan(ri);
        e = ri > e ? ri : e;
      }
    }
    if (bad) return JSH_ST_NAN;
    const bool rejected = e > 1.0;
    const double t_new = t + dt;
    if (!rejected && t_new == t) return JSH_ST_DT_UNDERFLOW;
    dt = next_dt(dt, e, rejected, 0.0);
    if (rejected) {
      C.rej++;
      if (++fails >= dp::FAIL_LIMIT) return JSH_ST_FAIL_LIMIT;
      continue;
    }
    fails = 0;
    C.acc++;
    x = y;
    k[0] = k[6];
    t = t_new;
  }
}

// The transfer of one hit ray at one frequency by the lanes of a group;
// lane 0 of the group gets the outputs.
template <bool FULL>
__device__ void transfer_item64(const JshModel& m, const JshPlane& pl, const JshParamsDev& Pp, const JshHit& hit,
                                double nu, int f, const Group64& G, ItemOut& o, Ctl64& tot) {
  uint32_t ev = 0;  // evaluation index of the item (random-direction key)
  o.tau = o.l = 0.0;
  o.iquv[0] = o.iquv[1] = o.iquv[2] = o.iquv[3] = 0.0;
  o.status = (uint32_t)hit.status | JSH_ST_HIT;
  const int64_t max_steps = Pp.max_steps > 0 ? Pp.max_steps : ((int64_t)1 << 22);
  D3 rd = d3(pl.dx, pl.dy, pl.dz);
  D3 rd2 = d3(pl.rx, pl.ry, pl.rz);
  D3 nl = rd * -1.;
  int nseg = hit.nseg;
  D3 cut = d3(0.0, 0.0, 0.0);  // where the last segment of the I / IQUV pass starts if tau_max cut it
  bool crossed = false;

  // ---- tau pass ----
  double background_tau = 0.0, thickness = 0.0;
  for (int sidx = 0; sidx < nseg; ++sidx) {
    D3 pin = d3(hit.seg[sidx][0], hit.seg[sidx][1], hit.seg[sidx][2]);
    D3 pout = d3(hit.seg[sidx][3], hit.seg[sidx][4], hit.seg[sidx][5]);
    D3 dd = pout - pin;
    double length = sqrt((dd.x * dd.x + dd.y * dd.y) + dd.z * dd.z);
    const Path64 P = path64(m, pin, rd, nl, nu, (uint32_t)hit.pix, (uint32_t)f);
    Ctl64 C{Pp.tau_atol, Pp.tau_rtol, Pp.dt_max, max_steps, 0, 0, 0};
    double x = 0.0, k[7], x_old = 0.0, dt_used = 0.0, t_old = 0.0;
    const uint32_t fail =
        tau_segment64(m, P, G, C, length, length / Pp.n, Pp.tau_max, ev, x, x_old, t_old, dt_used, k, crossed);
    tot.evals += C.evals;
    tot.acc += C.acc;
    tot.rej += C.rej;
    if (fail) {
      o.status |= fail;
      o.tau = background_tau + x;
      o.l = thickness + length;
      return;
    }
    if (crossed) {
      o.status |= JSH_ST_TAU_CROSSED;
      double t0 = t_old, t1 = t_old + dt_used, xm = x, t_m;
      const double ydiff = x - x_old;
      const double bspl = dt_used * k[0] - ydiff;
      const double r4 = ydiff - dt_used * k[6] - bspl;
      const double r5 = dt_used * (dp::D1 * k[0] + dp::D3 * k[2] + dp::D4 * k[3] + dp::D5 * k[4] + dp::D6 * k[5] +
                                   dp::D7 * k[6]);
      int it = 0;
      while (fabs(xm - Pp.tau_max) > Pp.tau_precision) {
        if (++it > 200) {
          o.status |= JSH_ST_BISECT_LIMIT;
          break;
        }
        t_m = 0.5 * (t0 + t1);
        double theta = (t_m - t_old) / dt_used, th1 = 1.0 - theta;
        xm = x_old + theta * (ydiff + th1 * (bspl + theta * (r4 + th1 * r5)));
        if (xm > Pp.tau_max) t1 = t_m;
        else t0 = t_m;
      }
      t_m = 0.5 * (t0 + t1);
      cut = pin + rd2 * t_m;
      nseg = sidx + 1;
    }
    background_tau += x;
    thickness += length;
    if (crossed) break;
  }
  o.tau = background_tau;
  o.l = thickness;
  if (!(background_tau > Pp.tau_min)) return;
  o.status |= JSH_ST_IQUV;

  // ---- I / IQUV pass ----
  double st = 0.0;
  for (int sidx = nseg - 1; sidx >= 0; --sidx) {
    D3 pin = d3(hit.seg[sidx][0], hit.seg[sidx][1], hit.seg[sidx][2]);
    D3 pout = crossed && sidx == nseg - 1 ? cut : d3(hit.seg[sidx][3], hit.seg[sidx][4], hit.seg[sidx][5]);
    D3 dd = pout - pin;
    double length = sqrt((dd.x * dd.x + dd.y * dd.y) + dd.z * dd.z);
    double auto_n = Pp.n;
    if (background_tau > 0.1) auto_n = steps_schedule(background_tau, Pp.n, 10 * Pp.n);
    const Path64 P = path64(m, pout, nl, nl, nu, (uint32_t)hit.pix, (uint32_t)f);
    Ctl64 C{Pp.atol, Pp.rtol, 0.0, max_steps, 0, 0, 0};
    const uint32_t fail = iquv_segment64<FULL>(m, P, G, C, length, length / auto_n, ev, st);
    tot.evals += C.evals;
    tot.acc += C.acc;
    tot.rej += C.rej;
    if (fail) {
      o.status |= fail;
      break;
    }
  }
  if (FULL) {
#pragma unroll
    for (int i = 0; i < 4; ++i) o.iquv[i] = from_lane(G, st, i);
  } else {
    o.iquv[0] = st;
  }
}

}  // namespace jsh
