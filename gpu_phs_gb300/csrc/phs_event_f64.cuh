// phs_event_f64.cuh -- one event of the forward map in FP64 (device code shared by the
// FP64 kernel and, as the exact fallback near kinematic limits, by the FP32-pair kernel).
//
// Arithmetic follows the reference CPU path (phs_cpu.cpp), whose expression order it keeps
// with separately rounded products and sums wherever a value feeds the kinematic ok test
// (msq mappings, the Kallen function and the mass sums), so ok flags match the reference
// bit for bit whenever the transcendental functions agree; factors and boosts use FMA.
//
// The FP64 pipe bounds this code (two lanes a cycle and SM), so the walk is written for few
// FP64 instructions:
//   * what can run beside the pipe does: the elementary functions, square roots and
//     reciprocals (phs_fix.h), halvings and doublings, the comparisons of the kinematic test;
//   * sums and products alone are FMAs with register constants (FxRegs: 16 cycles, not 19);
//   * a visit's frame step has a form per position in the tree (PHS_KIND_*), so that known
//     zeros cost nothing, and a visit of two outgoing daughters computes their momenta in its
//     own rest frame and takes them through its parent's frame, with no frame of its own;
//   * with massless daughters the Kallen function needs no product or square root, and two
//     of them need no 1/m, beta or gamma either: gamma E = E_b/2, beta gamma E = p_b/2;
//   * blocks that a visit skips are real branches: the compiler turns short ones into
//     predicated instructions, which take their turn on the FP64 pipe all the same.
// A tt event takes 302 FP64 instructions (445 before, 81 of them predicated off), the pipe is
// 91 % busy.  Against the library's functions and the plain product of matrices: 1e7 tt events
// 13.84 -> 8.29 (functions) -> 5.21 ms; 3e6 events of the 13 TeV caterpillar 0.346 -> 0.225,
// 2^22 events over 64 channels 1.10 -> 0.57, 5e5 tt events with their own beams 0.936 -> 0.416,
// 3e5 12-particle events 0.502 -> 0.216 ms (the first, second and last of these four with the
// pre-test's own changes).
// Momenta are nearer the exact map (median error of tt 3.1e-16 -> 2.2e-16 of the energy, against
// an 80-bit evaluation).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "phs_device.h"
#include "phs_fix.h"
#include "phs_math.h"
#include "phs_program.h"

#define PHS_PI 3.14159265358979323846
#define PHS_TWOPI2 39.47841760435743447534
#define PHS_TWOPI5 9792.62991312900650440772
#define PHS_STATE 20  // doubles per saved frame: L[16], msq, m, p, E

namespace {


__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }

// The STEP maps: calls, as they are rare and their library functions and divisions would be
// much of the kernels' code.
struct StepMap {
  double msq, f, aux;
};
__device__ __noinline__ StepMap map_msq_step(int t, double x, double s, double msq_min,
                                             double msq_max, double a0, double a1, double a2) {
  StepMap r;
  double z;
  if (t == PHS_MAP_STEP_H) {
    const double am = dsub(a0, x);
    z = dadd(dsub(a1 / am, a1 / a0), dmul(a2, x));
    r.f = (a1 / (am * am) + a2) * (msq_max - msq_min) / s;
    r.aux = 0.0;
  } else {
    const double tmp = dmul(exp(dmul(-x, a0) / a2), dadd(1.0, a1));
    z = dmul(-a2, log(dsub(tmp, a1)));
    r.f = a0 / (1.0 - a1 / tmp) * (msq_max - msq_min) / s;
    r.aux = tmp;
  }
  r.msq = dadd(dmul(z, msq_max), dmul(dsub(1.0, z), msq_min));
  return r;
}

// msq from x (phs_cpu.cpp:12-61), same expression order, no contraction.  f receives the
// mapping's factor without its constant part (a2; the range over s of the uniform map: the
// caller's, PhsChannel::f0 for uniform beams).  aux receives the mapping's transcendental
// term for the adjoint's derivatives: tan z (Breit-Wigner), the exponential term a0 exp(.)
// (collinear, infrared, radiation, t/u channel), exp(.)(1 + a1) (STEP_E); 0 otherwise.
__device__ __forceinline__ void map_msq(const FxRegs &k, int t, double x, double s, double m,
                                        double w, double msq_min, double msq_max, double a0,
                                        double a1, double a2, double &msq, double &f, double &aux) {
  aux = 0.0;
  switch (t) {
    case PHS_MAP_NO:
      msq = fx_add(k, fx_mul(k, fx_sub(k, k.one, x), msq_min), fx_mul(k, x, msq_max));
      f = 1.0;
      break;
    case PHS_MAP_SCHANNEL: {
      const double z = fx_add(k, fx_mul(k, fx_sub(k, k.one, x), a0), fx_mul(k, x, a1));
      // |z| < pi / 2, as integers (NaN is not)
      if ((fx_bits(z) & 0x7fffffffffffffffull) < 0x3ff921fb54442d18ull) {
        const double tz = fx_tan(z);
        msq = fx_mul(k, m, fx_add(k, fx_mul(k, w, tz), m));
        f = fma(tz, tz, k.one);
        aux = tz;
      } else {
        msq = 0.0;
        f = 0.0;
      }
      break;
    }
    case PHS_MAP_COLLINEAR:
    case PHS_MAP_INFRARED:
    case PHS_MAP_RADIATION: {
      const double msq1 = fx_mul(k, a0, fx_exp(fx_mul(k, x, a1)));
      msq = fx_add(k, fx_sub(k, msq1, a0), msq_min);
      f = msq1;
      aux = msq1;
      break;
    }
    case PHS_MAP_TCHANNEL:
    case PHS_MAP_UCHANNEL: {
      // one exponential per lane: the side of x = 0.5 selects its argument and the sum
      const bool lower = fx_gt(0.5, x);
      const double msq1 = fx_mul(k, a0, fx_exp(fx_mul(k, lower ? x : fx_sub(k, k.one, x), a1)));
      const double d = fx_sub(k, msq1, a0);
      msq = fx_add(k, lower ? d : fx_neg(d), lower ? msq_min : msq_max);
      f = msq1;
      aux = msq1;
      break;
    }
    case PHS_MAP_STEP_H:
    case PHS_MAP_STEP_E: {
      const StepMap r = map_msq_step(t, x, s, msq_min, msq_max, a0, a1, a2);
      msq = r.msq;
      f = r.f;
      aux = r.aux;
      break;
    }
    default:
      msq = 0.0;
      f = 0.0;
  }
}

// cos(theta) from x (phs_cpu.cpp:112-146).  The collinear branch keeps the reference's
// rounding: sin(theta) = sqrt(1 - ct^2) is ill-conditioned as |ct| -> 1.  The uniform map keeps
// the bits of ct = 1 - tmp and st = sqrt(tmp (2 - tmp)), tmp = 2 (1 - x): with 1 - x rounded, tmp
// and ct are exact, and so tmp (2 - tmp) = 1 - ct^2 is one FMA.  (sqrt(4 x (1 - x)) is an addition
// less and nearer to sin(theta) of x itself, but below x ~ 1e-3 it is another number than the
// reference's, and the derivatives divide by it: 3e-12 between the gradients of 1e6 WW events.)
__device__ __forceinline__ void map_ct(const FxRegs &k, int ct_class, double x, double b0,
                                       double b1, double &ct, double &st, double &f) {
  if (ct_class == PHS_CT_COLLINEAR) {
    const bool lower = fx_gt(0.5, x);
    const double y = lower ? x : fx_sub(k, k.one, x);
    const double tmp = fx_mul(k, b0, fx_exp(fx_mul(k, fx_scale(y, 1), b1)));
    const double d = fx_sub(k, tmp, b0);
    ct = fx_sub(k, lower ? d : fx_neg(d), lower ? k.one : fx_neg(k.one));
    if (ct >= -1.0 && ct <= 1.0) {
      st = fx_sqrt(fx_sub(k, k.one, fx_mul(k, ct, ct)), k);
      f = fx_mul(k, tmp, b1);
    } else {
      ct = 1.0;
      st = 0.0;
      f = 0.0;
    }
  } else {
    ct = fx_sub(k, k.one, fx_scale(fx_sub(k, k.one, x), 1));
    st = fx_sqrt(fma(-ct, ct, k.one), k);
    f = 1.0;
  }
}

// Rotation taking the z axis onto the direction of (bx, by, bz) about the axis z x b
// (Rodrigues), row-major 3x3: the friend boost's rotation (phs.cu:753-781 restated; the
// reference's matrix equals this one whenever by = 0, which holds for friends on the root's
// daughters, the only ones Whizard's trees carry).  The symmetric part is written as
// cos + (1 - cos) k k^T with k k^T from the transverse components, as the reference does:
// the form cos + sin^2/(1 + cos) turns rounding of the normalisation into errors of order
// eps/(1 + cos) as the axis approaches -z.  An axis exactly along -z (where the reference
// divides 0 by 0) gives the rotation by pi about x.
__device__ __forceinline__ void rot_z_onto(double bx, double by, double bz, double R[9]) {
  const double n = sqrt(bx * bx + by * by + bz * bz);
  bx /= n;
  by /= n;
  bz /= n;
  const double t = bx * bx + by * by;
  double r00 = 1.0, r01 = 0.0, r11 = bz;
  if (t > 0.0) {
    const double w = (1.0 - bz) / t;
    r00 = bz + w * (by * by);
    r01 = -w * (bx * by);
    r11 = bz + w * (bx * bx);
  }
  R[0] = r00; R[1] = r01; R[2] = bx;
  R[3] = r01; R[4] = r11; R[5] = by;
  R[6] = -bx; R[7] = -by; R[8] = bz;
}

// The channel's phase-space volume at sqrt(s) (phs_cpu.cpp:194-213), bottom-up in post-order
// with the reference's operation order: for the per-event-beam paths.  The divisions by
// the two constants are the correctly rounded corrected products (phs_div_by_const): the
// same bits.
__device__ __forceinline__ double channel_volume(const PhsChannel &ch, double sqrts) {
  double vol[PHS_MAX_VISITS];
  constexpr double c_int = 4 * PHS_TWOPI2, c_root = 4 * PHS_TWOPI5;
  constexpr double r_int = 1.0 / c_int, r_root = 1.0 / c_root;
  for (int i = 0; i < ch.n_vol; i++) {
    int k1 = ch.vol_child[i][0], k2 = ch.vol_child[i][1];
    double v1 = k1 >= 0 ? vol[k1] : 1.0, v2 = k2 >= 0 ? vol[k2] : 1.0;
    vol[i] = ch.vol_is_root[i] ? phs_div_by_const(dmul(v1, v2), c_root, r_root)
                               : phs_div_by_const(dmul(dmul(dmul(v1, v2), sqrts), sqrts), c_int, r_int);
  }
  return vol[ch.n_vol - 1];
}

// Mapping constants at one sqrt(s) (phs_cpu.cpp:452-531), for the per-event-beam path.
// inv_s = 1/s of the event.  The reference divides a2 by s and the Breit-Wigner argument by
// m w; here they are products with 1/s (once per event) and the compiled 1/(m w), within an
// ulp of the quotients (a2 weights the factor; a1 = atan(u) at u >= 10^3 moves by ulp/u).
// msq_min = m_min^2 and m^2 do not depend on sqrt(s): the compiled values (the same bits).
__device__ void child_constants(const FxRegs &k, const PhsChild &C, double sqrts, double m_tot,
                                double inv_s, double &a0, double &a1, double &a2,
                                double &msq_min, double &msq_max, double &m_max) {
  double m = C.m, w = C.w, m_min = C.m_min;
  m_max = fx_add(k, fx_sub(k, sqrts, m_tot), m_min);
  msq_min = C.msq_min;
  msq_max = fx_mul(k, m_max, m_max);
  a0 = a1 = a2 = 0.0;
  switch (C.map_id) {
    case PHS_MAP_NO:
      a1 = fx_sub(k, msq_max, msq_min);
      a2 = fx_mul(k, a1, inv_s);
      break;
    case PHS_MAP_SCHANNEL: {
      // a0 = atan((msq_min - m^2) / (m w)) does not depend on sqrt(s): the compiled
      // program's value (the host's atan of the same argument bits, as the reference's CPU
      // path computes it) serves every event
      a0 = C.a0;
      const double u = fx_mul(k, fx_sub(k, msq_max, C.msq0), C.inv_mw);
      if (!fx_gt(1024.0, u)) {   // phs_atan_large in the walk's forms (u >= 10^3 in practice)
        const double r = fx_rcp(u, k), r2 = fx_mul(k, r, r);
        const double at = fma(fx_mul(k, r, r2), fma(r2, 0.2, -1.0 / 3.0), r);
        a1 = (PHS_PIO2_HI - at) + PHS_PIO2_LO;
      } else {
        a1 = fx_lib_atan2(u, 1.0);
      }
      a2 = fx_mul(k, fx_mul(k, fx_sub(k, a1, a0), fx_mul(k, m, w)), inv_s);
      break;
    }
    case PHS_MAP_RADIATION:
    case PHS_MAP_COLLINEAR:
    case PHS_MAP_INFRARED: {
      double msq0 = C.map_id == PHS_MAP_RADIATION ? dmul(w, w) : dmul(m, m);
      a0 = msq0;
      a1 = log(dadd(dsub(msq_max, msq_min) / msq0, 1.0));
      a2 = a1 * inv_s;
      break;
    }
    case PHS_MAP_TCHANNEL:
    case PHS_MAP_UCHANNEL: {
      double msq0 = dmul(m, m);
      a0 = msq0;
      a1 = dmul(2.0, log(dadd(dsub(msq_max, msq_min) / dmul(2.0, msq0), 1.0)));
      a2 = a1 * inv_s;
      break;
    }
    case PHS_MAP_STEP_E: {
      double r = dmul(dmul(2.0, m), w) / dsub(msq_max, msq_min);
      a2 = r > 0.01 ? r : 0.01;
      a1 = exp(-(dsub(dmul(m, m), msq_min)) / dsub(msq_max, msq_min) / a2);
      a0 = dsub(1.0, dmul(a2, log(dadd(1.0, dmul(a1, exp(1.0 / a2))) / dadd(1.0, a1))));
      break;
    }
    case PHS_MAP_STEP_H: {
      a2 = dsub(dmul(m, m), msq_min) / dsub(msq_max, msq_min);
      double q = dmul(dmul(2.0, m), w) / dsub(msq_max, msq_min);
      double r = dmul(q, q) / a2;
      a1 = r > 0.000001 ? r : 0.000001;
      a0 = dadd(1.0, sqrt(dadd(1.0, dmul(4.0, a1) / dsub(1.0, a2)))) / 2.0;
      break;
    }
  }
}

__device__ __noinline__ double lib_sinpi(double x) { return sinpi(x); }
__device__ __noinline__ double lib_cospi(double x) { return cospi(x); }

// sin and cos of 2 pi x for a phi mapping's x: in fixed point for 0 <= x < 1, else the library's.
__device__ __forceinline__ void sincos2pi(double x, double &s, double &c) {
  if (fx_hi(x) < 0x3ff00000u) {
    fx_sincos2pi(x, s, c);
  } else {
    s = lib_sinpi(2.0 * x);
    c = lib_cospi(2.0 * x);
  }
}

// 1 / m and 1 / (2 m) of the visited branch's mass; 0 where m is not positive (its event
// fails the kinematic test).
__device__ __forceinline__ void mass_reciprocals(const FxRegs &k, double m, double &rm, double &hm) {
  rm = fx_hi(m) - 1u < 0x7fefffffu ? fx_rcp(m, k) : 0.0;
  hm = fx_scale(rm, -1);
}

// The Kallen function of the visited branch with the kinematic test, in the reference's
// rounding: sl = sqrt(lambda); `massless` has bit j set for a massless outgoing daughter j.
// With one of them lambda is d^2 and its rounded square root |d| itself (no over- or
// underflow for 2^-500 < |d| < 2^500; other d take the general form).  The test's upper
// bound, m <= m_max, is the caller's (per internal daughter, as its mass is formed).
__device__ __forceinline__ bool kallen_ok(const FxRegs &k, int massless, double msq_b, double m_b,
                                          const double cmsq[2], const double cm[2], double &sl) {
  double d = msq_b, msum = cm[0];
  if (massless == 0) {
    d = fx_sub(k, fx_sub(k, d, cmsq[0]), cmsq[1]);
    msum = fx_add(k, cm[0], cm[1]);
  } else if (massless != 3) {
    d = fx_sub(k, d, massless & 1 ? cmsq[1] : cmsq[0]);
    msum = massless & 1 ? cm[1] : cm[0];
  }
  bool positive;
  if (massless != 0 && (fx_hi(d) & 0x7fffffffu) - 0x20b00000u < 0x3e800000u) {
    sl = fx_from_bits(fx_bits(d) & 0x7fffffffffffffffull);
    positive = true;
  } else {
    const double lda = fx_sub(k, fx_mul(k, d, d), fx_mul(k, fx_scale(cmsq[0], 2), cmsq[1]));
    sl = fx_sqrt(lda, k);
    positive = fx_gt(lda, 0.0);
  }
  return positive && fx_gt(m_b, msum);
}

// Frame stack slot k of depth `depth`: one column per thread of a BLOCK-thread block.
template <int BLOCK>
__device__ __forceinline__ void stack_store(double *smem, int depth, int k, double v) {
  smem[(depth * PHS_STATE + k) * BLOCK + threadIdx.x] = v;
}
template <int BLOCK>
__device__ __forceinline__ double stack_load(const double *smem, int depth, int k) {
  return smem[(depth * PHS_STATE + k) * BLOCK + threadIdx.x];
}

// One event: segment `seg`, local index `local` (< seg.ev_count).  smem is this block's
// frame stack, PHS_STATE * stack_depth doubles per thread of a BLOCK-thread block.
// Checked build (phs_check.h): the event's channel, its whole x row, momentum row and event
// entries, and its program's visit count, before anything is read or written.
__device__ __forceinline__ bool event_in_bounds(const PhsLaunch &a, const PhsSegment &seg,
                                                int64_t local, int n_out, int n_visits) {
  const int64_t xrow = seg.x_base + local * seg.x_stride;
  const int64_t prow = seg.p_base + local * 4 * (int64_t)n_out;
  const int64_t ev = seg.ev_begin + local;
  return phs_in(local, seg.ev_count, PHS_CHK_EVENT) && phs_in(xrow, a.x_len, PHS_CHK_X) &&
         phs_in(xrow + seg.x_stride - 1, a.x_len, PHS_CHK_X) && phs_in(prow, a.p_len, PHS_CHK_P) &&
         phs_in(prow + 4 * (int64_t)n_out - 1, a.p_len, PHS_CHK_P) &&
         phs_in(ev, a.ev_len, PHS_CHK_EVENT) && phs_in(seg.factor_col, a.factor_stride, PHS_CHK_EVENT) &&
         phs_in(n_visits - 1, PHS_MAX_VISITS, PHS_CHK_VISITS);
}

// x[k] of an event row (checked build: k within the row; 0 otherwise).
__device__ __forceinline__ double xrow_at(const double *xe, int k, int stride) {
  return phs_in(k, stride, PHS_CHK_X) ? xe[k] : 0.0;
}

// A leaf's momentum row.
__device__ __forceinline__ void put_momentum(double *out, int index, int n_out, double q0, double q1,
                                             double q2, double q3) {
  if (!phs_in(index, n_out, PHS_CHK_P)) return;
  double2 *o = reinterpret_cast<double2 *>(out + 4 * index);
  o[0] = make_double2(q0, q1);
  o[1] = make_double2(q2, q3);
}

// The frame steps.  L is the parent's frame on entry and the visited branch's on return:
// L B_z(bg, ga) R_z(phi) R_y(theta), the boost along z first and the two rotations after it
// (phs_cpu.cpp:299-330 multiplies the same matrices), row by row in place: 12 FP64
// instructions for a full row where the product with the multiplied-out matrix takes 12 and
// 8 more to form its entries.
struct Step {
  double bg, ga, cp, sp, ct, st;
};
// Row (l0 l1 l2 l3); Z0: l0 = 0, Z2: l2 = 0.
template <bool Z0, bool Z2>
__device__ __forceinline__ void frame_row(const FxRegs &k, const Step &t, double *l) {
  const double n0 = Z0 ? fx_mul(k, l[3], t.bg) : fma(l[0], t.ga, fx_mul(k, l[3], t.bg));
  const double z = Z0 ? fx_mul(k, l[3], t.ga) : fma(l[0], t.bg, fx_mul(k, l[3], t.ga));
  const double u = Z2 ? fx_mul(k, t.cp, l[1]) : fma(t.sp, l[2], fx_mul(k, t.cp, l[1]));
  const double w = Z2 ? fx_mul(k, -t.sp, l[1]) : fma(t.cp, l[2], fx_mul(k, -t.sp, l[1]));
  l[0] = n0;
  l[1] = fma(t.ct, u, fx_mul(k, -t.st, z));
  l[2] = w;
  l[3] = fma(t.st, u, fx_mul(k, t.ct, z));
}

// The friend boost (phs.cu:853-910): the decay angles are measured from the friend beam's
// direction in the branch's rest frame, B_z(-bg) L^-1 (1, 0, 0, ff) (only its direction
// matters, so the lab boost inside L needs no special case); the step's matrix is
// B_z(bg) diag(1, R_f R(theta, phi)).  Uniform per channel: no divergence.
__device__ __forceinline__ void friend_step(double ff, const Step &t, double L[16]) {
  const double u0 = L[0] - ff * L[12];
  double Rf[9];
  rot_z_onto(-(L[1] - ff * L[13]), -(L[2] - ff * L[14]), -t.bg * u0 - t.ga * (L[3] - ff * L[15]), Rf);
  const double A[9] = {t.ct * t.cp, -t.sp, t.st * t.cp, t.ct * t.sp, t.cp, t.st * t.sp, -t.st, 0.0, t.ct};
  double Q[9];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++)
      Q[3 * r + c] = Rf[3 * r] * A[c] + Rf[3 * r + 1] * A[3 + c] + Rf[3 * r + 2] * A[6 + c];
  const double E1r[4] = {t.ga, t.bg * Q[6], t.bg * Q[7], t.bg * Q[8]};
  const double E2r[4] = {0.0, Q[0], Q[1], Q[2]};
  const double E3r[4] = {0.0, Q[3], Q[4], Q[5]};
  const double E4r[4] = {t.bg, t.ga * Q[6], t.ga * Q[7], t.ga * Q[8]};
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const double l0 = L[4 * r], l1 = L[4 * r + 1], l2 = L[4 * r + 2], l3 = L[4 * r + 3];
#pragma unroll
    for (int c = 0; c < 4; c++)
      L[4 * r + c] = l0 * E1r[c] + l1 * E2r[c] + l2 * E3r[c] + l3 * E4r[c];
  }
}

template <bool PER_EVENT, int BLOCK = PHS_FWD_BLOCK>
__device__ __forceinline__ void phs_event_f64(const PhsLaunch &a, const FxRegs &k,
                                              const PhsSegment &seg, int64_t local, double *smem) {
  if (!phs_in(seg.channel, a.n_programs, PHS_CHK_CHANNEL)) return;
  const PhsChannel &ch = a.channels[seg.channel];
  if (!event_in_bounds(a, seg, local, ch.n_out, ch.n_visits)) return;
  const int64_t ev = seg.ev_begin + local;
  const double *xe = a.x + seg.x_base + local * seg.x_stride;
  double *out = a.p + seg.p_base + local * 4 * (int64_t)ch.n_out;

  double sqrts = ch.sqrts;
  double lab_bg = ch.lab_bg, lab_ga = ch.lab_gamma;
  const bool lab = PER_EVENT || ch.lab != 0;
  if (PER_EVENT) {
    const double E1 = a.E1[ev], E2 = a.E2[ev];
    const double r = fx_sqrt(fx_mul(k, E1, E2), k);
    sqrts = fx_add(k, r, r);
    lab_bg = fx_div(fx_sub(k, E1, E2), sqrts, k);
    lab_ga = fx_sqrt(fma(lab_bg, lab_bg, k.one), k);
  }
  const double s = fx_mul(k, sqrts, sqrts);
  const double inv_s = PER_EVENT ? fx_rcp(s, k) : 0.0;   // per-event mapping constants

  // frame of the visited branch (the root's parent frame, the lab boost or 1, is in its step)
  double L[16];
#pragma unroll
  for (int i = 0; i < 16; i++) L[i] = 0.0;
  double msq_b = s, m_b = sqrts, p_b = 0.0, E_b = sqrts;
  double factor = PER_EVENT ? 1.0 : ch.f0;
  bool ok = true;
  int sp = 0, halved = 0;

  const int n_visits = ch.n_visits;
  for (int v = 0; v < n_visits; v++) {
    const PhsVisit &V = ch.visit[v];
    const int4 head = *reinterpret_cast<const int4 *>(&V.code);   // (code, child_code)
    const int code = head.x;
    double cmsq[2] = {V.child[0].msq_leaf, V.child[1].msq_leaf}, cm[2] = {V.child[0].m_leaf, V.child[1].m_leaf};
    // (not unrolled: the mapping code of one daughter serves both)
#pragma unroll 1
    for (int j = 0; j < 2; j++) {
      const PhsChild &C = V.child[j];
      const int cc = j == 0 ? head.y : head.z, map_id = cc >> 1 & 15;
      if (cc & 1) {
        double mq, mj;
        double a0 = C.a0, a1 = C.a1, a2 = C.a2, mn = C.msq_min, mx = C.msq_max, mmax = C.m_max;
        if (PER_EVENT) child_constants(k, C, sqrts, ch.m_tot, inv_s, a0, a1, a2, mn, mx, mmax);
        double f, aux;
        map_msq(k, map_id, xrow_at(xe, cc >> 8 & 0xff, seg.x_stride), s, C.m, C.w, mn, mx, a0, a1, a2,
                mq, f, aux);
        if (PER_EVENT && map_id != PHS_MAP_STEP_E && map_id != PHS_MAP_STEP_H) factor = fx_mul(k, factor, a2);
        if (map_id != PHS_MAP_NO) factor = fx_mul(k, factor, f);
        mj = fx_sqrt(mq, k);
        ok = ok && !fx_gt(mj, mmax);   // NaN fails at the daughter's own visit
        if (j == 0) {
          cmsq[0] = mq;
          cm[0] = mj;
        } else {
          cmsq[1] = mq;
          cm[1] = mj;
        }
      }
    }
    // Kallen function and kinematic test at the visited branch (phs_cpu.cpp:218-233)
    const int massless = code >> 18 & 3;
    double sl;
    ok = kallen_ok(k, massless, msq_b, m_b, cmsq, cm, sl) && ok;
    // one reciprocal of m serves p_decay = sqrt(lda)/(2m), sqrt(lda)/m^2, bg, gamma and the
    // daughters' energies E = (m^2 + m_j^2 - m_k^2)/(2m) (the two-body energy, equal to the
    // reference's sqrt(m_j^2 + p^2)); a massless daughter's is p, the other's then m - p.
    // Two massless daughters share m equally, their sqrt(lda)/m^2 is 1, and as the last
    // visit of their line nothing else needs 1/m.  sqrt(lda)/m^2 is kept halved, the powers
    // of two put back at the end.
    int kind = code >> 20 & 7;
    if (lab)
      kind = kind == PHS_KIND_ROOT ? PHS_KIND_ROOT_LAB
             : kind == PHS_KIND_FIRST ? PHS_KIND_FIRST_LAB
             : kind == PHS_KIND_LEAVES_FIRST ? PHS_KIND_LEAVES : kind;
    const bool pair = kind == PHS_KIND_LEAVES || kind == PHS_KIND_LEAVES_FIRST;
    double rm = 0.0, pc, ce0, ce1;
    if (massless == 3) {
      pc = ce0 = ce1 = fx_scale(m_b, -1);
      if (!pair) rm = fx_hi(m_b) - 1u < 0x7fefffffu ? fx_rcp(m_b, k) : 0.0;   // a friend's, or n_out = 2
    } else {
      double hm;
      if (!PER_EVENT && (code >> 17 & 1)) {
        rm = ch.inv_sqrts;
        hm = fx_scale(rm, -1);
      } else {
        mass_reciprocals(k, m_b, rm, hm);
      }
      pc = fx_mul(k, sl, hm);
      factor = fx_mul(k, factor, fx_mul(k, pc, rm));
      halved++;
      if (massless == 0) {
        const double dc = fx_sub(k, cmsq[0], cmsq[1]);
        ce0 = fx_mul(k, fx_add(k, msq_b, dc), hm);
        ce1 = fx_mul(k, fx_sub(k, msq_b, dc), hm);
      } else {
        const double eo = fx_sub(k, m_b, pc);
        ce0 = massless & 1 ? pc : eo;
        ce1 = massless & 1 ? eo : pc;
      }
    }

    // the decay angles
    Step t;
    sincos2pi(xrow_at(xe, code & 0xff, seg.x_stride), t.sp, t.cp);
    double b0 = V.b0, b1 = V.b1;
    if (PER_EVENT && (code >> 16 & 1) == PHS_CT_COLLINEAR) {
      b0 = dmul(V.m, V.m) / s;
      b1 = log(dadd(b0, 1.0) / b0);
    }
    double fct;
    map_ct(k, (code >> 16 & 1), xrow_at(xe, code >> 8 & 0xff, seg.x_stride), b0, b1, t.ct, t.st, fct);
    if ((code >> 16 & 1) == PHS_CT_COLLINEAR) factor = fx_mul(k, factor, fct);   // the uniform map's factor is 1

    if (pair) {
      // two outgoing daughters: (E, 0, 0, +-p) rotated by (theta, phi), boosted along z by
      // (bg, gamma) and taken through the parent's frame; the transverse part is shared up
      // to its sign
      const double pst = fx_mul(k, pc, t.st), qx = fx_mul(k, pst, t.cp), qy = fx_mul(k, pst, t.sp);
      double qa0, qa3, qb0, qb3;   // daughters 0 and 1 along t and z
      if (massless == 3) {
        const double eh = fx_scale(E_b, -1), ph = fx_scale(p_b, -1);
        qa0 = fma(ph, t.ct, eh);
        qb0 = fma(-ph, t.ct, eh);
        qa3 = fma(eh, t.ct, ph);
        qb3 = fma(-eh, t.ct, ph);
      } else {
        const double bg = fx_mul(k, p_b, rm), ga = fx_mul(k, E_b, rm), qz = fx_mul(k, pc, t.ct);
        const double z0 = fx_mul(k, bg, qz), z3 = fx_mul(k, ga, qz);
        qa0 = fma(ga, ce0, z0);
        qb0 = fma(ga, ce1, -z0);
        qa3 = fma(bg, ce0, z3);
        qb3 = fma(bg, ce1, -z3);
      }
      double qa[4], qb[4];
      if (kind == PHS_KIND_LEAVES_FIRST) {
        // the parent's frame is the root's rotation: (1,0,0,0) (0,*,*,*) (0,*,*,*) (0,*,0,*)
        qa[0] = qa0;
        qb[0] = qb0;
#pragma unroll
        for (int r = 1; r < 4; r++) {
          const double l1 = L[4 * r + 1], l2 = L[4 * r + 2], l3 = L[4 * r + 3];
          const double w = r < 3 ? fma(l2, qy, fx_mul(k, l1, qx)) : fx_mul(k, l1, qx);
          qa[r] = fma(l3, qa3, w);
          qb[r] = fma(l3, qb3, -w);
        }
      } else {
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const double l0 = L[4 * r], l1 = L[4 * r + 1], l2 = L[4 * r + 2], l3 = L[4 * r + 3];
          const double w = fma(l2, qy, fx_mul(k, l1, qx));
          qa[r] = fma(l0, qa0, fma(l3, qa3, w));
          qb[r] = fma(l0, qb0, fma(l3, qb3, -w));
        }
      }
      put_momentum(out, head.y >> 16, ch.n_out, qa[0], qa[1], qa[2], qa[3]);
      put_momentum(out, head.z >> 16, ch.n_out, qb[0], qb[1], qb[2], qb[3]);
    } else {
      // rotation + boost of the visited branch (phs_cpu.cpp:299-330)
      if (!(code >> 17 & 1)) {
        t.bg = fx_mul(k, p_b, rm);
        t.ga = fx_mul(k, E_b, rm);
      }
      switch (kind) {
        case PHS_KIND_ROOT:
          // parent frame and boost are the identity: the rotation alone
          L[0] = 1.0;  L[1] = 0.0;                       L[2] = 0.0;          L[3] = 0.0;
          L[4] = 0.0;  L[5] = fx_mul(k, t.ct, t.cp);     L[6] = fx_neg(t.sp); L[7] = fx_mul(k, t.st, t.cp);
          L[8] = 0.0;  L[9] = fx_mul(k, t.ct, t.sp);     L[10] = t.cp;        L[11] = fx_mul(k, t.st, t.sp);
          L[12] = 0.0; L[13] = fx_neg(t.st);             L[14] = 0.0;         L[15] = t.ct;
          break;
        case PHS_KIND_ROOT_LAB:
          // behind the lab boost B_z(lab_bg): rows 1 and 2 as above
          L[0] = lab_ga;  L[1] = fx_mul(k, -lab_bg, t.st);  L[2] = 0.0;          L[3] = fx_mul(k, lab_bg, t.ct);
          L[4] = 0.0;     L[5] = fx_mul(k, t.ct, t.cp);     L[6] = fx_neg(t.sp); L[7] = fx_mul(k, t.st, t.cp);
          L[8] = 0.0;     L[9] = fx_mul(k, t.ct, t.sp);     L[10] = t.cp;        L[11] = fx_mul(k, t.st, t.sp);
          L[12] = lab_bg; L[13] = fx_mul(k, -lab_ga, t.st); L[14] = 0.0;         L[15] = fx_mul(k, lab_ga, t.ct);
          break;
        case PHS_KIND_FIRST:
          // row 0 of the root's rotation is (1, 0, 0, 0)
          L[0] = t.ga;
          L[1] = fx_mul(k, -t.st, t.bg);
          L[2] = 0.0;
          L[3] = fx_mul(k, t.ct, t.bg);
          frame_row<true, false>(k, t, L + 4);
          frame_row<true, false>(k, t, L + 8);
          frame_row<true, true>(k, t, L + 12);
          break;
        case PHS_KIND_FIRST_LAB:
          // the root's frame with the lab boost: entries (0,2), (1,0), (2,0), (3,2) are 0
          frame_row<false, true>(k, t, L);
          frame_row<true, false>(k, t, L + 4);
          frame_row<true, false>(k, t, L + 8);
          frame_row<false, true>(k, t, L + 12);
          break;
        case PHS_KIND_FRIEND:
          friend_step((double)V.friend_sign, t, L);
          break;
        default:
#pragma unroll
          for (int r = 0; r < 4; r++) frame_row<false, false>(k, t, L + 4 * r);
      }
      // leaf momenta: L_new * (E, 0, 0, +-p) (phs_cpu.cpp:286-291).  (A loop that is not
      // unrolled: the compiler would issue the FP64 instructions of an absent leaf too.)
#pragma unroll 1
      for (int j = head.y & 1 ? (head.z & 1 ? 2 : 1) : 0; j < 2; j++) {
        const int cc = j == 0 ? head.y : head.z;
        if (cc & 1) break;
        const double E = j == 0 ? ce0 : ce1, pj = j == 0 ? pc : fx_neg(pc);
        double q[4];
#pragma unroll
        for (int r = 0; r < 4; r++) q[r] = fma(L[4 * r], E, fx_mul(k, L[4 * r + 3], pj));
        put_momentum(out, cc >> 16, ch.n_out, q[0], q[1], q[2], q[3]);
      }
    }

    // next frame: push one internal child, carry the other (or pop)
    // (selects instead of indexing keep the child values in registers)
    const int push = (code >> 25 & 3) - 1, carry = (code >> 23 & 3) - 1;
    if (push >= 0 && phs_in(sp, a.stack_depth, PHS_CHK_STACK)) {
      const bool j0 = push == 0;
#pragma unroll
      for (int i = 0; i < 16; i++) stack_store<BLOCK>(smem, sp, i, L[i]);
      stack_store<BLOCK>(smem, sp, 16, j0 ? cmsq[0] : cmsq[1]);
      stack_store<BLOCK>(smem, sp, 17, j0 ? cm[0] : cm[1]);
      stack_store<BLOCK>(smem, sp, 18, j0 ? pc : fx_neg(pc));
      stack_store<BLOCK>(smem, sp, 19, j0 ? ce0 : ce1);
      sp++;
    }
    if (carry >= 0) {
      const bool j0 = carry == 0;
      msq_b = j0 ? cmsq[0] : cmsq[1];
      m_b = j0 ? cm[0] : cm[1];
      p_b = j0 ? pc : fx_neg(pc);
      E_b = j0 ? ce0 : ce1;
    } else if (sp > 0) {
      sp--;
#pragma unroll
      for (int i = 0; i < 16; i++) L[i] = stack_load<BLOCK>(smem, sp, i);
      msq_b = stack_load<BLOCK>(smem, sp, 16);
      m_b = stack_load<BLOCK>(smem, sp, 17);
      p_b = stack_load<BLOCK>(smem, sp, 18);
      E_b = stack_load<BLOCK>(smem, sp, 19);
    }
  }

  a.volume[ev] = PER_EVENT ? channel_volume(ch, sqrts) : ch.volume;
  a.factor[ev * a.factor_stride + seg.factor_col] =
      ok ? fx_mul(k, factor, fx_double((1023u + halved) << 20, 0u)) : 0.0;
  a.ok[ev] = ok ? 1 : 0;
  if (!ok) {
    double2 *o = reinterpret_cast<double2 *>(out);
    for (int i = 0; i < 2 * ch.n_out; i++) o[i] = make_double2(0.0, 0.0);
  }
}


// Pass A of the compacting kernels: the kinematic test of one event alone -- the msq
// mappings of its internal branches and the Kallen / mass tests of phs_event_f64 in the
// same arithmetic, so the flag is the same bit -- without angles or boosts.  An event that
// fails gets its outputs here (momenta 0, factor 0, ok 0, the channel volume); one that
// passes gets them from phs_event_f64 in pass B.  Returns ok.  smem: the event's frame
// stack (only the msq and m slots are used).
template <bool PER_EVENT, int BLOCK = PHS_FWD_BLOCK>
__device__ __forceinline__ bool phs_ok_f64(const PhsLaunch &a, const FxRegs &k,
                                           const PhsSegment &seg, int64_t local, double *smem) {
  if (!phs_in(seg.channel, a.n_programs, PHS_CHK_CHANNEL)) return false;
  const PhsChannel &ch = a.channels[seg.channel];
  if (!event_in_bounds(a, seg, local, ch.n_out, ch.n_visits)) return false;
  const int64_t ev = seg.ev_begin + local;
  const double *xe = a.x + seg.x_base + local * seg.x_stride;
  double sqrts = ch.sqrts;
  if (PER_EVENT) {
    const double r = fx_sqrt(fx_mul(k, a.E1[ev], a.E2[ev]), k);
    sqrts = fx_add(k, r, r);
  }
  const double s = fx_mul(k, sqrts, sqrts);
  const double inv_s = PER_EVENT ? fx_rcp(s, k) : 0.0;   // per-event mapping constants
  double msq_b = s, m_b = sqrts;
  bool ok = true;
  int sp = 0;
  const int n_visits = ch.n_visits;
  for (int v = 0; v < n_visits; v++) {
    const PhsVisit &V = ch.visit[v];
    const int4 head = *reinterpret_cast<const int4 *>(&V.code);   // (code, child_code)
    const int code = head.x;
    double cmsq[2] = {V.child[0].msq_leaf, V.child[1].msq_leaf}, cm[2] = {V.child[0].m_leaf, V.child[1].m_leaf};
    // (not unrolled: the mapping code of one daughter serves both)
#pragma unroll 1
    for (int j = 0; j < 2; j++) {
      const PhsChild &C = V.child[j];
      const int cc = j == 0 ? head.y : head.z, map_id = cc >> 1 & 15;
      if (cc & 1) {
        double mq, mj;
        double a0 = C.a0, a1 = C.a1, a2 = C.a2, mn = C.msq_min, mx = C.msq_max, mmax = C.m_max;
        if (PER_EVENT) child_constants(k, C, sqrts, ch.m_tot, inv_s, a0, a1, a2, mn, mx, mmax);
        double f, aux;
        map_msq(k, map_id, xrow_at(xe, cc >> 8 & 0xff, seg.x_stride), s, C.m, C.w, mn, mx, a0, a1, a2,
                mq, f, aux);
        mj = fx_sqrt(mq, k);
        ok = ok && !fx_gt(mj, mmax);
        if (j == 0) {
          cmsq[0] = mq;
          cm[0] = mj;
        } else {
          cmsq[1] = mq;
          cm[1] = mj;
        }
      }
    }
    double sl;
    ok = kallen_ok(k, code >> 18 & 3, msq_b, m_b, cmsq, cm, sl) && ok;
    const int push = (code >> 25 & 3) - 1, carry = (code >> 23 & 3) - 1;
    if (push >= 0 && phs_in(sp, a.stack_depth, PHS_CHK_STACK)) {
      const bool j0 = push == 0;
      stack_store<BLOCK>(smem, sp, 16, j0 ? cmsq[0] : cmsq[1]);
      stack_store<BLOCK>(smem, sp, 17, j0 ? cm[0] : cm[1]);
      sp++;
    }
    if (carry >= 0) {
      const bool j0 = carry == 0;
      msq_b = j0 ? cmsq[0] : cmsq[1];
      m_b = j0 ? cm[0] : cm[1];
    } else if (sp > 0) {
      sp--;
      msq_b = stack_load<BLOCK>(smem, sp, 16);
      m_b = stack_load<BLOCK>(smem, sp, 17);
    }
  }
  if (!ok) {
    a.volume[ev] = PER_EVENT ? channel_volume(ch, sqrts) : ch.volume;
    a.factor[ev * a.factor_stride + seg.factor_col] = 0.0;
    a.ok[ev] = 0;
    double2 *o = reinterpret_cast<double2 *>(a.p + seg.p_base + local * 4 * (int64_t)ch.n_out);
    for (int i = 0; i < 2 * ch.n_out; i++) o[i] = make_double2(0.0, 0.0);
  }
  return ok;
}

// The split forms' claim numbering: tile[s] = sum over the segments before s of ceil(count / 32),
// tile[n] the total.  Up to PHS_INLINE_SEGS segments every block of the walk forms it from the
// pre-test's counts in shared memory (a launch for it, and one for its counters, took 5 us of a
// call); more come from phs_count_scan_kernel.  Collective over the block.
__device__ __forceinline__ const int64_t *claim_numbering(const PhsLaunch &a, int64_t *shared) {
  if (a.n_segments > PHS_INLINE_SEGS) return a.pass_tile;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int64_t carry = 0;
    for (int base = 0; base < a.n_segments; base += 32) {
      const int s = base + lane;
      const int64_t v = s < a.n_segments ? ((int64_t)a.pass_count[s] + 31) / 32 : 0;
      int64_t inc = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (s < a.n_segments) shared[s] = carry + inc - v;
      carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) shared[a.n_segments] = carry;
  }
  __syncthreads();
  return shared;
}

// The persistent loop of the compacting kernels.  Each warp runs pass A on its 32-event
// tiles (`pass_a(seg, local)` tests an event, writes it if it fails, and returns whether it
// passed) and appends the passing events to its queue in shared memory (q: 64 slots);
// pass B (`pass_b(seg_index, seg, local)`, collective, the full event or none: local < 0) drains the queue 32 events at a time with
// every lane busy.  The queue holds events of one segment only, so the visit program stays
// warp-uniform: a tile of another segment first drains it.  Pass A and pass B have one
// call site each, which keeps the (large) event code once in the kernel.
//
// Work is claimed in chunks of CHUNK consecutive tiles of one segment: CHUNK = 1 (single
// tiles), or a.chunk_tiles (CHUNK = 0; PhsSegment::chunk_begin; a segment's last chunk may be
// shorter), whichever was measured faster for the kernel.  With a.work set, a warp claims
// its next chunk from that counter when it finishes one (events of different channels and
// kinematics cost very different amounts, and static shares leave SMs idle at the end);
// without, chunks are strided over the grid.
template <int CHUNK, class PassA, class PassB>
__device__ __forceinline__ void compacting_loop(const PhsLaunch &a, int64_t *q, PassA pass_a,
                                                PassB pass_b) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const PhsSegment *segs = a.n_segments <= PHS_INLINE_SEGS ? a.seg_inline : a.segments;
  int64_t claimed = 0;
  auto next_chunk = [&]() -> int64_t {
    if (a.work) {
      unsigned long long c = 0;
      if (lane == 0) c = atomicAdd(a.work, 1ull);
      return (int64_t)__shfl_sync(0xffffffffu, c, 0);
    }
    return warp0 + (claimed++) * n_warps;
  };
  int qn = 0, qseg = 0;  // warp-uniform: queue length and its segment
  int cseg = 0;          // segment of the current chunk
  int64_t tile = 0, tile_end = 0;
  bool done = false;
  static_assert(CHUNK == 1 || CHUNK == 0, "chunks of 1 or a.chunk_tiles tiles");
  auto claim = [&]() {
    const int64_t c = next_chunk();
    done = c >= (CHUNK == 1 ? a.n_tiles : a.n_chunks);
    if (done) return;
    int lo = 0, hi = a.n_segments - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((CHUNK == 1 ? segs[mid].tile_begin : segs[mid].chunk_begin) <= c) lo = mid; else hi = mid - 1;
    }
    cseg = lo;
    if (CHUNK == 1) {
      tile = c;
      tile_end = c + 1;
      return;
    }
    const int64_t seg_tiles = (segs[lo].ev_count + 31) / 32;
    tile = segs[lo].tile_begin + (c - segs[lo].chunk_begin) * a.chunk_tiles;
    const int64_t end = tile + a.chunk_tiles, seg_end = segs[lo].tile_begin + seg_tiles;
    tile_end = end < seg_end ? end : seg_end;
  };
  claim();
  for (;;) {
    bool passed = false;
    int64_t local = 0;
    if (!done) {
      local = (tile - segs[cseg].tile_begin) * 32 + lane;
      if (local < segs[cseg].ev_count) passed = pass_a(segs[cseg], local);
    }
    const unsigned m = __ballot_sync(0xffffffffu, passed);
    // stage 0: drain the queue (end of the work, or a new segment); 1: append; 2: drain
    // full warps
    int stage = (done || (m != 0 && qn > 0 && qseg != cseg)) ? 0 : 1;
    for (;;) {
      int take;
      if (stage == 0) {
        if (qn == 0) { stage = 1; continue; }
        take = qn < 32 ? qn : 32;
      } else if (stage == 1) {
        if (m != 0) {
          const int slot = qn + __popc(m & ((1u << lane) - 1u));
          if (passed && phs_in(slot, 64, PHS_CHK_QUEUE)) q[slot] = local;
          qn += __popc(m);
          qseg = cseg;
        }
        stage = 2;
        continue;
      } else {
        if (qn < 32) break;
        take = 32;
      }
      __syncwarp();
      const int64_t l = lane < take && phs_in(qn - take + lane, 64, PHS_CHK_QUEUE) ? q[qn - take + lane] : -1;
      __syncwarp();
      qn -= take;
      pass_b(qseg, segs[qseg], l);
    }
    if (done) break;
    if (++tile == tile_end) claim();
  }
}

}  // namespace
