// phs_adjoint.cu -- reverse-mode derivatives of the forward map (FP64).
//
// For cotangents pbar (of the momenta) and jbar (of the log-Jacobian log(factor)), one
// thread per event computes
//     xbar[k]      = sum pbar . dp/dx_k + jbar dlogJ/dx_k                 (every x)
//     thbar[b][0/1] = the same for d/dm and d/dGamma of Breit-Wigner branch b
// (b = the branch's msq x index).  Two passes per event:
//   1. the forward walk of phs_event_f64.cuh recomputed, keeping only the state each visit
//      starts from (msq, m, p, E of the visited branch) and the frame current before each
//      pop -- no per-branch matrices;
//   2. the visits in reverse.  A visit's frame step is a boost along z and two rotations
//      applied to each row of the frame (frame_row, phs_event_f64.cuh); the reverse walk
//      undoes them row by row in place, which recovers the parent's frame, and takes the
//      row's adjoint back through the same three steps: 30 FP64 instructions a row with the
//      adjoints of both angles and the rapidity, where the 4x4 matrices took 44.  Adjoints of
//      frames travel up the tree with a stack that mirrors the forward one.
// A visit of two outgoing daughters has no frame of its own: their momenta are the parent's
// frame times two vectors (phs_event_f64), differentiated as such.
// The FP64 pipe bounds it (77 % busy with 8 warps a SM; block sizes of 32 to 128 threads and
// 9 or 10 warps gave the same times): 1e6 tt events 3.37 ms with matrices and library functions,
// 2.94 ms with the forward walk's functions, 1.66 ms in this form (1410 -> 835 FP64
// instructions an event).
// Of a branch's kinematics (its msq, mass, momentum and energy in the parent's frame) the
// independent ones are msq and the momentum, so an internal daughter hands two adjoints to
// its parent.
// Friend (beam-axis) visits rotate the decay frame onto an axis computed from the parent
// frame; the forward pass keeps that axis per visit, and the reverse walk rebuilds the
// rotation and differentiates it (a forward-mode evaluation with three tangents).
// Uniform beams only.  Events with ok = 0 get zero derivatives.
//
// STORED instantiations are the stored-matrix form for comparison: the forward pass writes
// every visit's parent frame (16 doubles per visit and event) to a device buffer, as the
// reference keeps its per-event boost chain in device memory (Ld, 16 N_BOOSTS doubles per
// event, phs.cu:1421-1422), and the reverse walk reads the parent frames back instead of
// recovering them with the inverse boost.  Same derivatives up to rounding; it costs the
// buffer (n_events x max_visits x 128 bytes) and its HBM traffic.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "phs_device.h"
#include "phs_event_f64.cuh"
#include "phs_program.h"

#define PHS_ADJ_BLOCK 64
#define PHS_ADJ_STATE 6    // per visit: msq, m, p, E of the visited branch, sqrt(lambda), 1/m
#define PHS_ADJ_ANG 6      // per visit: cos phi, sin phi, ct, st, the ct map's factor, and the
                           // visited branch's msq map term (aux of map_msq)
#define PHS_ADJ_FRAME 18   // adjoint stack entry: Lbar[16], msqbar, pbar

namespace {

struct AdjLayout {
  int state0, ang0, pop0, stack0;  // offsets (in slots) of the per-thread regions
  int fr0;                               // friend visits: the rotation axis, 3 per visit
  int nv, npops, depth;                  // visits, pop frames and stack depth the regions hold
};

// A value with its derivatives along three directions (forward-mode differentiation).
struct D3 {
  double v, d[3];
};
__device__ __forceinline__ D3 d3(double v, int k) {
  D3 r = {v, {0.0, 0.0, 0.0}};
  if (k >= 0) r.d[k] = 1.0;
  return r;
}
__device__ __forceinline__ D3 operator+(D3 a, D3 b) {
  return {a.v + b.v, {a.d[0] + b.d[0], a.d[1] + b.d[1], a.d[2] + b.d[2]}};
}
__device__ __forceinline__ D3 operator-(D3 a, D3 b) {
  return {a.v - b.v, {a.d[0] - b.d[0], a.d[1] - b.d[1], a.d[2] - b.d[2]}};
}
__device__ __forceinline__ D3 operator-(D3 a) { return {-a.v, {-a.d[0], -a.d[1], -a.d[2]}}; }
__device__ __forceinline__ D3 operator*(D3 a, D3 b) {
  return {a.v * b.v, {a.d[0] * b.v + a.v * b.d[0], a.d[1] * b.v + a.v * b.d[1],
                      a.d[2] * b.v + a.v * b.d[2]}};
}
__device__ __forceinline__ D3 operator/(D3 a, D3 b) {
  const double q = a.v / b.v, r = 1.0 / b.v;
  return {q, {(a.d[0] - q * b.d[0]) * r, (a.d[1] - q * b.d[1]) * r, (a.d[2] - q * b.d[2]) * r}};
}
__device__ __forceinline__ D3 d3_sqrt(D3 a) {
  const double s = sqrt(a.v), h = 0.5 / s;
  return {s, {a.d[0] * h, a.d[1] * h, a.d[2] * h}};
}

// dR[i]/d(bx, by, bz) of rot_z_onto (same formula and branch): J[3 i + k].
__device__ __forceinline__ void rot_z_onto_jacobian(double bx0, double by0, double bz0,
                                                    double J[27]) {
  D3 bx = d3(bx0, 0), by = d3(by0, 1), bz = d3(bz0, 2);
  const D3 n = d3_sqrt(bx * bx + by * by + bz * bz);
  bx = bx / n;
  by = by / n;
  bz = bz / n;
  const D3 t = bx * bx + by * by;
  D3 r00 = d3(1.0, -1), r01 = d3(0.0, -1), r11 = bz;
  if (t.v > 0.0) {
    const D3 w = (d3(1.0, -1) - bz) / t;
    r00 = bz + w * (by * by);
    r01 = -(w * (bx * by));
    r11 = bz + w * (bx * bx);
  }
  const D3 R[9] = {r00, r01, bx, r01, r11, by, -bx, -by, bz};
#pragma unroll
  for (int i = 0; i < 9; i++)
#pragma unroll
    for (int k = 0; k < 3; k++) J[3 * i + k] = R[i].d[k];
}

// Q = R_f A(theta, phi), the friend visit's spatial rotation (phs_event_f64.cuh).
__device__ __forceinline__ void friend_rotation(const double Rf[9], double ct, double st,
                                                double cphi, double sphi, double Q[9]) {
  const double A[9] = {ct * cphi, -sphi, st * cphi, ct * sphi, cphi, st * sphi, -st, 0.0, ct};
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++)
      Q[3 * r + c] = Rf[3 * r] * A[c] + Rf[3 * r + 1] * A[3 + c] + Rf[3 * r + 2] * A[6 + c];
}

__device__ __forceinline__ double &slot(double *sm, int i) {
  return sm[i * PHS_ADJ_BLOCK + threadIdx.x];
}

// The msq mapping's derivatives at x, contracted with the adjoint of msq and jb, that of
// log(factor): xb, and for Breit-Wigner branches those in the mass and the width (through the
// atan bounds a0, a1 as well).  aux is the forward map's transcendental term (map_msq): tan z,
// a0 exp(.), or exp(.)(1 + a1).
__device__ __forceinline__ void map_adjoint(const FxRegs &k, const PhsChild &C, const PhsAdjChild &A,
                                            double x, double aux, double msqb, double jb, double &xb,
                                            double &mb, double &wb) {
  mb = wb = 0.0;
  switch (C.map_id) {
    case PHS_MAP_NO:
      xb = fx_mul(k, msqb, fx_sub(k, C.msq_max, C.msq_min));
      break;
    case PHS_MAP_SCHANNEL: {
      // msq = m^2 + m w t, log f = log a2 + log(1 + t^2), t = tan z, dt = (1 + t^2) dz: the
      // adjoint of z, then z = (1 - x) a0 + x a1 and the explicit terms
      const double t = aux, tj = fx_mul(k, fx_scale(t, 1), jb);
      const double zb = fma(fx_mul(k, A.mw, msqb), fma(t, t, k.one), tj), x1 = fx_sub(k, k.one, x);
      xb = fx_mul(k, zb, A.da);
      mb = fma(zb, fma(x, A.da1_dm, fx_mul(k, x1, A.da0_dm)),
               fma(msqb, fma(C.w, t, A.two_m), fx_mul(k, A.dlf_dm0, jb)));
      wb = fma(zb, fma(x, A.da1_dw, fx_mul(k, x1, A.da0_dw)),
               fma(msqb, fx_mul(k, C.m, t), fx_mul(k, A.dlf_dw0, jb)));
      break;
    }
    case PHS_MAP_COLLINEAR:
    case PHS_MAP_INFRARED:
    case PHS_MAP_RADIATION:
      xb = fx_mul(k, C.a1, fma(msqb, aux, jb));
      break;
    case PHS_MAP_TCHANNEL:
    case PHS_MAP_UCHANNEL:
      xb = fx_mul(k, C.a1, fma(msqb, aux, fx_gt(0.5, x) ? jb : fx_neg(jb)));
      break;
    case PHS_MAP_STEP_H: {
      const double q = C.a0 - x, g = C.a1 / (q * q) + C.a2;
      xb = msqb * ((C.msq_max - C.msq_min) * g) + jb * (2.0 * C.a1 / (q * q * q) / g);
      break;
    }
    case PHS_MAP_STEP_E:
      xb = msqb * (C.a0 * aux / (aux - C.a1) * (C.msq_max - C.msq_min)) +
           jb * (C.a0 * C.a1 / (C.a2 * (aux - C.a1)));
      break;
    default:
      xb = 0.0;
  }
}

// The adjoint of the ct map's x from that of theta (thb) and jb: dct/dx = 2 (uniform) or
// 2 fct (fct = b1 b0 exp(.), the collinear map's factor; 0 outside the mapped range, which is
// constant), dtheta = -dct / st, dlog fct/dx = +-2 b1.  ctb: the adjoint of ct, for st = 0 (x =
// 0), where st counts as constant.
__device__ __forceinline__ double ct_adjoint(const FxRegs &k, int ct_class, double x, double b1,
                                             double st, double fct, double thb, double ctb,
                                             double jb) {
  if (!fx_gt(st, 0.0)) return ct_class == PHS_CT_COLLINEAR ? 0.0 : fx_scale(ctb, 1);
  const double r = fx_mul(k, -thb, fx_rcp(st, k));
  if (ct_class != PHS_CT_COLLINEAR) return fx_scale(r, 1);
  return fx_scale(fma(r, fct, fx_mul(k, fx_gt(0.5, x) ? b1 : fx_neg(b1), jb)), 1);
}

// One row back through a frame step: n is the row of the visited branch's frame on entry and
// of the parent's on return, nb its adjoint; th, ph and et gather the adjoints of theta, phi
// and the rapidity.  (n1, n3) = R(theta)(u, z), (u, w) = R(phi)(l1, l2), (n0, z) = B(l0, l3).
__device__ __forceinline__ void adjoint_row(const FxRegs &k, const Step &t, double *n, double *nb,
                                            double &th, double &ph, double &et) {
  th = fma(nb[3], n[1], th);
  th = fma(-nb[1], n[3], th);
  const double u = fma(t.ct, n[1], fx_mul(k, t.st, n[3])), z = fma(t.ct, n[3], fx_mul(k, -t.st, n[1]));
  const double ub = fma(t.ct, nb[1], fx_mul(k, t.st, nb[3])), zb = fma(t.ct, nb[3], fx_mul(k, -t.st, nb[1]));
  const double w = n[2], wb = nb[2], n0 = n[0], nb0 = nb[0];
  ph = fma(ub, w, ph);
  ph = fma(-wb, u, ph);
  n[1] = fma(t.cp, u, fx_mul(k, -t.sp, w));
  n[2] = fma(t.cp, w, fx_mul(k, t.sp, u));
  nb[1] = fma(t.cp, ub, fx_mul(k, -t.sp, wb));
  nb[2] = fma(t.cp, wb, fx_mul(k, t.sp, ub));
  et = fma(nb0, z, et);
  et = fma(zb, n0, et);
  n[0] = fma(t.ga, n0, fx_mul(k, -t.bg, z));
  n[3] = fma(t.ga, z, fx_mul(k, -t.bg, n0));
  nb[0] = fma(t.ga, nb0, fx_mul(k, t.bg, zb));
  nb[3] = fma(t.ga, zb, fx_mul(k, t.bg, nb0));
}
// Row r of the same where the parent is the root without a lab boost: the parent's row is
// (1,0,0,0) for r = 0 and has l0 = 0 (r = 3: l2 = 0) else, and the root reads no adjoint of
// its column 0, of its row 0, or of its entry (3,2).
template <int R>
__device__ __forceinline__ void adjoint_row_first(const FxRegs &k, const Step &t, double *n, double *nb,
                                                  double &th, double &ph, double &et) {
  th = fma(nb[3], n[1], th);
  th = fma(-nb[1], n[3], th);
  const double zb = fma(t.ct, nb[3], fx_mul(k, -t.st, nb[1]));
  const double z = R == 0 ? t.bg : fma(t.ct, n[3], fx_mul(k, -t.st, n[1]));
  et = fma(nb[0], z, et);
  et = fma(zb, n[0], et);
  if (R == 0) {
    n[0] = 1.0;
    n[1] = n[2] = n[3] = 0.0;
    return;
  }
  const double u = fma(t.ct, n[1], fx_mul(k, t.st, n[3])), ub = fma(t.ct, nb[1], fx_mul(k, t.st, nb[3]));
  const double w = n[2], wb = nb[2];
  ph = fma(ub, w, ph);
  ph = fma(-wb, u, ph);
  n[1] = fma(t.cp, u, fx_mul(k, -t.sp, w));
  n[2] = R == 3 ? 0.0 : fma(t.cp, w, fx_mul(k, t.sp, u));
  n[3] = fma(t.ga, z, fx_mul(k, -t.bg, n[0]));
  n[0] = 0.0;
  nb[3] = fma(t.ga, zb, fx_mul(k, t.bg, nb[0]));
  nb[1] = fma(t.cp, ub, fx_mul(k, -t.sp, wb));
  nb[2] = R == 3 ? 0.0 : fma(t.cp, wb, fx_mul(k, t.sp, ub));
  nb[0] = 0.0;
}

// FRIENDS: the process has friend visits (a separate instantiation keeps their code out of
// the register allocation of the others).  STORED: the stored-matrix form (above); store
// holds frame slot (v * 16 + i) of event ev at store[(v * 16 + i) * store_events + ev].
template <bool FRIENDS, bool STORED>
__global__ void __launch_bounds__(PHS_ADJ_BLOCK)
    phs_adjoint_kernel(const __grid_constant__ PhsLaunch a, const PhsAdjChannel *__restrict__ adj,
                       const double *__restrict__ pbar, const double *__restrict__ jbar,
                       double *__restrict__ xbar, double *__restrict__ thbar, int th_stride,
                       AdjLayout lay, double *__restrict__ store, int64_t store_events) {
  extern __shared__ double sm[];
  const FxRegs kr = fx_regs();
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;

  for (int64_t tile = warp0; tile < a.n_tiles; tile += n_warps) {
    const PhsSegment *segs = a.n_segments <= PHS_INLINE_SEGS ? a.seg_inline : a.segments;
    int lo = 0, hi = a.n_segments - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (segs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    const PhsSegment seg = segs[lo];
    const int64_t local = (tile - seg.tile_begin) * 32 + lane;
    if (local >= seg.ev_count) continue;
    if (!phs_in(seg.channel, a.n_programs, PHS_CHK_CHANNEL)) continue;
    const PhsChannel &ch = a.channels[seg.channel];
    const PhsAdjChannel &ad = adj[seg.channel];
    // checked build: the rows of x, xbar (x's layout), pbar (p's) and thbar, and a program
    // that fits the shared-memory regions sized for it
    if (!event_in_bounds(a, seg, local, ch.n_out, ch.n_visits) ||
        !phs_in(ch.n_visits - 1, lay.nv, PHS_CHK_VISITS) ||
        !phs_in(ad.n_pops, lay.npops + 1, PHS_CHK_VISITS))
      continue;
    const int64_t ev = seg.ev_begin + local;
    const double *xe = a.x + seg.x_base + local * seg.x_stride;
    double *xb = xbar + seg.x_base + local * seg.x_stride;
    double *tb = thbar + ev * th_stride;
    const double *pb = pbar + seg.p_base + local * 4 * (int64_t)ch.n_out;
    const double jb = jbar ? jbar[ev] : 0.0;
    const double sqrts = ch.sqrts, s = fx_mul(kr, sqrts, sqrts);
    const bool lab = ch.lab != 0;
    const int n_visits = ch.n_visits;
    const auto kind_of = [&](const PhsVisit &V) {
      if (!lab) return V.kind;
      return V.kind == PHS_KIND_ROOT ? PHS_KIND_ROOT_LAB
             : V.kind == PHS_KIND_FIRST ? PHS_KIND_FIRST_LAB
             : V.kind == PHS_KIND_LEAVES_FIRST ? PHS_KIND_LEAVES : V.kind;
    };

    // ---------------------------------------------------------------- 1. forward walk
    double L[16];
#pragma unroll
    for (int i = 0; i < 16; i++) L[i] = 0.0;
    if (STORED) {
      L[0] = L[15] = lab ? ch.lab_gamma : 1.0;
      L[5] = L[10] = 1.0;
      L[3] = L[12] = lab ? ch.lab_bg : 0.0;
    }
    double msq_b = s, m_b = sqrts, p_b = 0.0, E_b = sqrts;
    bool ok = true;
    int sp = 0, np = 0;
    for (int v = 0; v < n_visits; v++) {
      const PhsVisit &V = ch.visit[v];
      if (STORED && phs_in(ev, store_events, PHS_CHK_STORE)) {
#pragma unroll
        for (int i = 0; i < 16; i++) store[(int64_t)(v * 16 + i) * store_events + ev] = L[i];
      }
      const int sb = lay.state0 + PHS_ADJ_STATE * v, ab = lay.ang0 + PHS_ADJ_ANG * v;
      slot(sm, sb + 0) = msq_b;
      slot(sm, sb + 1) = m_b;
      slot(sm, sb + 2) = p_b;
      slot(sm, sb + 3) = E_b;
      double cmsq[2] = {V.child[0].msq_leaf, V.child[1].msq_leaf}, cm[2] = {V.child[0].m_leaf, V.child[1].m_leaf};
#pragma unroll 1
      for (int j = 0; j < 2; j++) {
        const PhsChild &C = V.child[j];
        if (!C.internal) continue;
        double mq, f, aux;
        map_msq(kr, C.map_id, xrow_at(xe, C.x_msq, seg.x_stride), s, C.m, C.w, C.msq_min, C.msq_max, C.a0,
                C.a1, C.a2, mq, f, aux);
        const double mj = fx_sqrt(mq, kr);
        ok = ok && !fx_gt(mj, C.m_max);
        const int cv = ad.visit[v].child_visit[j];
        if (phs_in(cv, n_visits, PHS_CHK_VISITS)) slot(sm, lay.ang0 + PHS_ADJ_ANG * cv + 5) = aux;
        if (j == 0) {
          cmsq[0] = mq;
          cm[0] = mj;
        } else {
          cmsq[1] = mq;
          cm[1] = mj;
        }
      }
      const int massless = V.massless, kind = kind_of(V);
      const bool pair = kind == PHS_KIND_LEAVES || kind == PHS_KIND_LEAVES_FIRST;
      double sl, rm, hm;
      ok = kallen_ok(kr, massless, msq_b, m_b, cmsq, cm, sl) && ok;
      mass_reciprocals(kr, m_b, rm, hm);
      slot(sm, sb + 4) = sl;
      slot(sm, sb + 5) = rm;
      Step t;
      double fct;
      sincos2pi(xrow_at(xe, V.x_phi, seg.x_stride), t.sp, t.cp);
      map_ct(kr, V.ct_class, xrow_at(xe, V.x_ct, seg.x_stride), V.b0, V.b1, t.ct, t.st, fct);
      slot(sm, ab + 0) = t.cp;
      slot(sm, ab + 1) = t.sp;
      slot(sm, ab + 2) = t.ct;
      slot(sm, ab + 3) = t.st;
      slot(sm, ab + 4) = fct;
      if (!pair) {
        // (two outgoing daughters: the frame stays the parent's)
        const double pc = fx_mul(kr, sl, hm), dc = fx_sub(kr, cmsq[0], cmsq[1]);
        const double ce0 = fx_mul(kr, fx_add(kr, msq_b, dc), hm), ce1 = fx_mul(kr, fx_sub(kr, msq_b, dc), hm);
        t.bg = V.self_root ? 0.0 : fx_mul(kr, p_b, rm);
        t.ga = V.self_root ? 1.0 : fx_mul(kr, E_b, rm);
        switch (kind) {
          case PHS_KIND_ROOT:
          case PHS_KIND_ROOT_LAB: {
            const double lg = lab ? ch.lab_gamma : 1.0, lb = lab ? ch.lab_bg : 0.0;
            L[0] = lg;  L[1] = fx_mul(kr, -lb, t.st);   L[2] = 0.0;          L[3] = fx_mul(kr, lb, t.ct);
            L[4] = 0.0; L[5] = fx_mul(kr, t.ct, t.cp);  L[6] = fx_neg(t.sp); L[7] = fx_mul(kr, t.st, t.cp);
            L[8] = 0.0; L[9] = fx_mul(kr, t.ct, t.sp);  L[10] = t.cp;        L[11] = fx_mul(kr, t.st, t.sp);
            L[12] = lb; L[13] = fx_mul(kr, -lg, t.st);  L[14] = 0.0;         L[15] = fx_mul(kr, lg, t.ct);
            break;
          }
          case PHS_KIND_FIRST:
            L[0] = t.ga;
            L[1] = fx_mul(kr, -t.st, t.bg);
            L[2] = 0.0;
            L[3] = fx_mul(kr, t.ct, t.bg);
            frame_row<true, false>(kr, t, L + 4);
            frame_row<true, false>(kr, t, L + 8);
            frame_row<true, true>(kr, t, L + 12);
            break;
          case PHS_KIND_FRIEND:
            if (FRIENDS) {
              // L1 = B_z(bg) diag(1, R_f A(theta, phi)), R_f onto the friend beam's direction
              // in the branch's rest frame; the axis is kept for the reverse walk
              const double ff = V.friend_sign;
              const int fb = lay.fr0 + 3 * v;
              slot(sm, fb + 0) = -(L[1] - ff * L[13]);
              slot(sm, fb + 1) = -(L[2] - ff * L[14]);
              slot(sm, fb + 2) = -t.bg * (L[0] - ff * L[12]) - t.ga * (L[3] - ff * L[15]);
              friend_step(ff, t, L);
            }
            break;
          default:
#pragma unroll
            for (int r = 0; r < 4; r++) frame_row<false, false>(kr, t, L + 4 * r);
        }
        if (V.push >= 0 && phs_in(sp, lay.depth, PHS_CHK_STACK)) {
          const bool j0 = V.push == 0;
          const int base = lay.stack0 + PHS_STATE * sp;
#pragma unroll
          for (int i = 0; i < 16; i++) slot(sm, base + i) = L[i];
          slot(sm, base + 16) = j0 ? cmsq[0] : cmsq[1];
          slot(sm, base + 17) = j0 ? cm[0] : cm[1];
          slot(sm, base + 18) = j0 ? pc : fx_neg(pc);
          slot(sm, base + 19) = j0 ? ce0 : ce1;
          sp++;
        }
        if (V.carry >= 0) {
          const bool j0 = V.carry == 0;
          msq_b = j0 ? cmsq[0] : cmsq[1];
          m_b = j0 ? cm[0] : cm[1];
          p_b = j0 ? pc : fx_neg(pc);
          E_b = j0 ? ce0 : ce1;
        }
      }
      if (V.carry < 0 && sp > 0) {
        // the frame the reverse walk resumes with after this pop
        if (phs_in(np, lay.npops, PHS_CHK_STACK)) {
#pragma unroll
          for (int i = 0; i < 16; i++) slot(sm, lay.pop0 + 16 * np + i) = L[i];
        }
        np++;
        sp--;
        const int base = lay.stack0 + PHS_STATE * sp;
#pragma unroll
        for (int i = 0; i < 16; i++) L[i] = slot(sm, base + i);
        msq_b = slot(sm, base + 16);
        m_b = slot(sm, base + 17);
        p_b = slot(sm, base + 18);
        E_b = slot(sm, base + 19);
      }
    }
    // what no visit writes: x padding, and everything of an event that fails the test
    for (int i = ok ? ch.n_x_used : 0; i < seg.x_stride; i++) xb[i] = 0.0;
    for (int i = ok ? 2 * (ch.n_out - 2) : 0; i < th_stride; i++) tb[i] = 0.0;
    if (!ok) continue;

    // ---------------------------------------------------------------- 2. reverse walk
    // L holds the frame after the last visit; Lb the adjoint of the current visit's frame
    double Lb[16];
#pragma unroll
    for (int i = 0; i < 16; i++) Lb[i] = 0.0;
    double sb_msq = 0.0, sb_p = 0.0;  // carried daughter's msq and momentum adjoints
    int asp = 0;
    for (int v = n_visits - 1; v >= 0; v--) {
      const PhsVisit &V = ch.visit[v];
      const PhsAdjVisit &A = ad.visit[v];
      const int sb = lay.state0 + PHS_ADJ_STATE * v, ab = lay.ang0 + PHS_ADJ_ANG * v;
      const double msq_v = slot(sm, sb + 0), m_v = slot(sm, sb + 1), p_v = slot(sm, sb + 2);
      const double E_v = slot(sm, sb + 3);
      const int massless = V.massless, kind = kind_of(V);
      const bool pair = kind == PHS_KIND_LEAVES || kind == PHS_KIND_LEAVES_FIRST;
      double cmsq[2], c_msqb[2] = {0.0, 0.0}, c_pb[2] = {0.0, 0.0};
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const PhsChild &C = V.child[j];
        cmsq[j] = C.msq_leaf;
        if (C.internal)
          cmsq[j] = phs_in(A.child_visit[j], n_visits, PHS_CHK_VISITS)
                        ? slot(sm, lay.state0 + PHS_ADJ_STATE * A.child_visit[j]) : 1.0;
      }
      if (V.carry >= 0) {
        const bool j0 = V.carry == 0;
        c_msqb[0] = j0 ? sb_msq : 0.0;
        c_pb[0] = j0 ? sb_p : 0.0;
        c_msqb[1] = j0 ? 0.0 : sb_msq;
        c_pb[1] = j0 ? 0.0 : sb_p;
      }
      if (V.push >= 0 && phs_in(asp - 1, lay.depth, PHS_CHK_STACK)) {
        asp--;
        const int base = lay.stack0 + PHS_ADJ_FRAME * asp;
#pragma unroll
        for (int i = 0; i < 16; i++) Lb[i] = fx_add(kr, Lb[i], slot(sm, base + i));
        const double mq = slot(sm, base + 16), pq = slot(sm, base + 17);
        const bool j0 = V.push == 0;
        c_msqb[0] = j0 ? mq : c_msqb[0];
        c_pb[0] = j0 ? pq : c_pb[0];
        c_msqb[1] = j0 ? c_msqb[1] : mq;
        c_pb[1] = j0 ? c_pb[1] : pq;
      }
      // the visit's quantities (the square root and the reciprocal as the forward pass left them)
      const double sl = slot(sm, sb + 4), rm = slot(sm, sb + 5), hm = fx_scale(rm, -1);
      Step t;
      t.cp = slot(sm, ab + 0);
      t.sp = slot(sm, ab + 1);
      t.ct = slot(sm, ab + 2);
      t.st = slot(sm, ab + 3);
      t.bg = V.self_root ? 0.0 : fx_mul(kr, p_v, rm);
      t.ga = V.self_root ? 1.0 : fx_mul(kr, E_v, rm);
      double pc, ce0, ce1;
      if (massless == 3) {
        pc = ce0 = ce1 = fx_scale(m_v, -1);
      } else {
        pc = fx_mul(kr, sl, hm);
        const double dc = fx_sub(kr, cmsq[0], cmsq[1]);
        ce0 = fx_mul(kr, fx_add(kr, msq_v, dc), hm);
        ce1 = fx_mul(kr, fx_sub(kr, msq_v, dc), hm);
      }
      // adjoints of theta, phi and the rapidity, of p_decay and the daughters' energies
      double th = 0.0, ph = 0.0, et = 0.0, pcb = 0.0, ceb0 = 0.0, ceb1 = 0.0;
      double ct0b = 0.0;             // of cos(theta), where sin(theta) = 0
      double Eb = 0.0, pb_v = 0.0;   // of the branch's own energy and momentum (massless pairs)
      if (pair) {
        // P0 = L (qa0, qx, qy, qa3), P1 = L (qb0, -qx, -qy, qb3) (phs_event_f64), L the parent's
        // frame: its adjoint and those of the vectors' components
        const double pst = fx_mul(kr, pc, t.st), qx = fx_mul(kr, pst, t.cp), qy = fx_mul(kr, pst, t.sp);
        const double eh = fx_scale(E_v, -1), hp = fx_scale(p_v, -1), qz = fx_mul(kr, pc, t.ct);
        double qa0, qa3, qb0, qb3;
        if (massless == 3) {
          qa0 = fma(hp, t.ct, eh);
          qb0 = fma(-hp, t.ct, eh);
          qa3 = fma(eh, t.ct, hp);
          qb3 = fma(-eh, t.ct, hp);
        } else {
          const double z0 = fx_mul(kr, t.bg, qz), z3 = fx_mul(kr, t.ga, qz);
          qa0 = fma(t.ga, ce0, z0);
          qb0 = fma(t.ga, ce1, -z0);
          qa3 = fma(t.bg, ce0, z3);
          qb3 = fma(t.bg, ce1, -z3);
        }
        const bool in = phs_in(V.child[0].out_index, ch.n_out, PHS_CHK_ADJ) && phs_in(V.child[1].out_index, ch.n_out, PHS_CHK_ADJ);
        const double *Pa = pb + 4 * (in ? V.child[0].out_index : 0), *Pb = pb + 4 * (in ? V.child[1].out_index : 0);
        double a0b = 0.0, b0b = 0.0, a3b = 0.0, b3b = 0.0, xq = 0.0, yq = 0.0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const double pa = Pa[r], pbr = Pb[r], d = fx_sub(kr, pa, pbr);
          a0b = fma(pa, L[4 * r], a0b);
          b0b = fma(pbr, L[4 * r], b0b);
          a3b = fma(pa, L[4 * r + 3], a3b);
          b3b = fma(pbr, L[4 * r + 3], b3b);
          xq = fma(d, L[4 * r + 1], xq);
          yq = fma(d, L[4 * r + 2], yq);
          Lb[4 * r + 0] = fma(pa, qa0, fx_mul(kr, pbr, qb0));
          Lb[4 * r + 1] = fx_mul(kr, d, qx);
          Lb[4 * r + 2] = fx_mul(kr, d, qy);
          Lb[4 * r + 3] = fma(pa, qa3, fx_mul(kr, pbr, qb3));
        }
        const double d0 = fx_sub(kr, a0b, b0b), d3 = fx_sub(kr, a3b, b3b);
        const double pstb = fma(xq, t.cp, fx_mul(kr, yq, t.sp));
        ph = fma(yq, qx, fx_mul(kr, -xq, qy));
        double ctb;
        if (massless == 3) {
          Eb = fx_scale(fma(t.ct, d3, fx_add(kr, a0b, b0b)), -1);
          pb_v = fx_scale(fma(t.ct, d0, fx_add(kr, a3b, b3b)), -1);
          ctb = fma(hp, d0, fx_mul(kr, eh, d3));
          pcb = fx_mul(kr, pstb, t.st);
        } else {
          const double gab = fma(a0b, ce0, fma(b0b, ce1, fx_mul(kr, d3, qz)));
          const double bgb = fma(a3b, ce0, fma(b3b, ce1, fx_mul(kr, d0, qz)));
          et = fma(gab, t.bg, fx_mul(kr, bgb, t.ga));
          ceb0 = fma(a0b, t.ga, fx_mul(kr, a3b, t.bg));
          ceb1 = fma(b0b, t.ga, fx_mul(kr, b3b, t.bg));
          const double qzb = fma(t.bg, d0, fx_mul(kr, t.ga, d3));
          ctb = fx_mul(kr, qzb, pc);
          pcb = fma(qzb, t.ct, fx_mul(kr, pstb, t.st));
        }
        ct0b = ctb;
        // theta from ct and st
        th = fma(fx_mul(kr, pstb, pc), t.ct, fx_mul(kr, -t.st, ctb));
      } else {
        // leaf daughters: P_j = L (ce_j, 0, 0, +-pc)
#pragma unroll 1
        for (int j = V.child[0].internal ? (V.child[1].internal ? 2 : 1) : 0; j < 2; j++) {
          const PhsChild &C = V.child[j];
          if (C.internal) break;
          if (!phs_in(C.out_index, ch.n_out, PHS_CHK_ADJ)) continue;
          const double ce = j == 0 ? ce0 : ce1, pj = j == 0 ? pc : fx_neg(pc);
          const double *P = pb + 4 * C.out_index;
          double v0 = 0.0, v3 = 0.0;
#pragma unroll
          for (int r = 0; r < 4; r++) {
            const double q = P[r];
            Lb[4 * r + 0] = fma(q, ce, Lb[4 * r + 0]);
            Lb[4 * r + 3] = fma(q, pj, Lb[4 * r + 3]);
            v0 = fma(L[4 * r], q, v0);
            v3 = fma(L[4 * r + 3], q, v3);
          }
          if (j == 0) {
            ceb0 = v0;
            pcb = fx_add(kr, pcb, v3);
          } else {
            ceb1 = v0;
            pcb = fx_sub(kr, pcb, v3);
          }
        }
        // an internal daughter's momentum is +-p_decay (its energy follows from it)
        pcb = fx_add(kr, pcb, fx_sub(kr, c_pb[0], c_pb[1]));
#pragma unroll 1
        for (int q = fx_gt(t.st, 0.0) ? 1 : 0; q < 1; q++) {   // (a loop: a real branch)
#pragma unroll
          for (int r = 0; r < 16; r += 4) ct0b = fma(t.ct, fma(Lb[r + 1], L[r + 1], Lb[r + 3] * L[r + 3]), ct0b);
        }
        if (FRIENDS && kind == PHS_KIND_FRIEND) {
          // L1 = F = B_z(bg) diag(1, Q), Q = R_f(axis) A(theta, phi), axis from the parent frame
          // (kept by the forward pass).  L_pre = L eta F^T eta, Lpre_bar = Lb F^T,
          // Fbar = L_pre^T Lb, then through Q to the angles, R_f and the axis, and from the axis
          // back to the parent frame, bg and gamma.
          const double ct = t.ct, st = t.st, cphi = t.cp, sphi = t.sp, bg = t.bg, ga = t.ga;
          const double eta[4] = {1.0, -1.0, -1.0, -1.0};
          double Lp[16], Lpb[16];
          const double ff = V.friend_sign;
          const int fb = lay.fr0 + 3 * v;
          const double ax = slot(sm, fb + 0), ay = slot(sm, fb + 1), az = slot(sm, fb + 2);
          double Rf[9], Q[9];
          rot_z_onto(ax, ay, az, Rf);
          friend_rotation(Rf, ct, st, cphi, sphi, Q);
          const double F[16] = {ga,  bg * Q[6], bg * Q[7], bg * Q[8],
                                0.0, Q[0],      Q[1],      Q[2],
                                0.0, Q[3],      Q[4],      Q[5],
                                bg,  ga * Q[6], ga * Q[7], ga * Q[8]};
#pragma unroll
          for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
              double acc = 0.0, accb = 0.0;
#pragma unroll
              for (int k = 0; k < 4; k++) {
                if ((c == 1 || c == 2) && k == 0) continue;  // F's zeros
                acc += L[4 * r + k] * (eta[k] * eta[c]) * F[4 * c + k];
                accb += Lb[4 * r + k] * F[4 * c + k];
              }
              Lp[4 * r + c] = acc;
              Lpb[4 * r + c] = accb;
            }
          double Fb[16];
#pragma unroll
          for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
              double acc = 0.0;
#pragma unroll
              for (int k = 0; k < 4; k++) acc += Lp[4 * k + r] * Lb[4 * k + c];
              Fb[4 * r + c] = acc;
            }
          double gab = Fb[0] + Fb[13] * Q[6] + Fb[14] * Q[7] + Fb[15] * Q[8];
          double bgb = Fb[12] + Fb[1] * Q[6] + Fb[2] * Q[7] + Fb[3] * Q[8];
          double Qb[9];
#pragma unroll
          for (int c = 0; c < 3; c++) {
            Qb[c] = Fb[5 + c];
            Qb[3 + c] = Fb[9 + c];
            Qb[6 + c] = bg * Fb[1 + c] + ga * Fb[13 + c];
          }
          // Q = R_f A: Abar = R_f^T Qbar, R_f bar = Qbar A^T
          const double Am[9] = {ct * cphi, -sphi, st * cphi, ct * sphi, cphi, st * sphi, -st, 0.0, ct};
          double Ab[9], Rb[9];
#pragma unroll
          for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
              Ab[3 * i + j] = Rf[i] * Qb[j] + Rf[3 + i] * Qb[3 + j] + Rf[6 + i] * Qb[6 + j];
              Rb[3 * i + j] = Qb[3 * i] * Am[3 * j] + Qb[3 * i + 1] * Am[3 * j + 1] + Qb[3 * i + 2] * Am[3 * j + 2];
            }
          const double ctb = Ab[0] * cphi + Ab[3] * sphi + Ab[8];
          const double stb = Ab[2] * cphi + Ab[5] * sphi - Ab[6];
          const double cpb = Ab[0] * ct + Ab[2] * st + Ab[4];
          const double spb = -Ab[1] + Ab[3] * ct + Ab[5] * st;
          // R_f(axis): axis bar = J^T R_f bar
          double J[27];
          rot_z_onto_jacobian(ax, ay, az, J);
          double axb[3] = {0.0, 0.0, 0.0};
#pragma unroll
          for (int i = 0; i < 9; i++)
#pragma unroll
            for (int k = 0; k < 3; k++) axb[k] += Rb[i] * J[3 * i + k];
          // axis = (-(Lp01 - ff Lp31), -(Lp02 - ff Lp32), -bg u0 - gamma (Lp03 - ff Lp33)),
          // u0 = Lp00 - ff Lp30
          const double u0 = Lp[0] - ff * Lp[12];
          Lpb[1] -= axb[0];
          Lpb[13] += ff * axb[0];
          Lpb[2] -= axb[1];
          Lpb[14] += ff * axb[1];
          Lpb[0] -= bg * axb[2];
          Lpb[12] += ff * bg * axb[2];
          Lpb[3] -= ga * axb[2];
          Lpb[15] += ff * ga * axb[2];
          bgb -= u0 * axb[2];
          gab -= (Lp[3] - ff * Lp[15]) * axb[2];
          et = gab * bg + bgb * ga;
          th = ct * stb - st * ctb;
          ph = cphi * spb - sphi * cpb;
#pragma unroll
          for (int i = 0; i < 16; i++) {
            L[i] = Lp[i];
            Lb[i] = Lpb[i];
          }
        } else {
          switch (kind) {
            case PHS_KIND_ROOT:
            case PHS_KIND_ROOT_LAB:
              // the parent frame is fixed (1 or the lab boost), and so is the root's own boost:
              // u and w are (cos phi, -sin phi), (sin phi, cos phi) in rows 1, 2, else 0
#pragma unroll
              for (int r = 0; r < 4; r++) {
                th = fma(Lb[4 * r + 3], L[4 * r + 1], th);
                th = fma(-Lb[4 * r + 1], L[4 * r + 3], th);
                if (r == 0 || r == 3) continue;
                const double ub = fma(t.ct, Lb[4 * r + 1], fx_mul(kr, t.st, Lb[4 * r + 3]));
                ph = fma(ub, r == 1 ? -t.sp : t.cp, ph);
                ph = fma(-Lb[4 * r + 2], r == 1 ? t.cp : t.sp, ph);
              }
              break;
            case PHS_KIND_FIRST:
              adjoint_row_first<0>(kr, t, L, Lb, th, ph, et);
              adjoint_row_first<1>(kr, t, L + 4, Lb + 4, th, ph, et);
              adjoint_row_first<2>(kr, t, L + 8, Lb + 8, th, ph, et);
              adjoint_row_first<3>(kr, t, L + 12, Lb + 12, th, ph, et);
              break;
            default:
#pragma unroll
              for (int r = 0; r < 4; r++) adjoint_row(kr, t, L + 4 * r, Lb + 4 * r, th, ph, et);
          }
        }
        if (STORED && phs_in(ev, store_events, PHS_CHK_STORE)) {
#pragma unroll
          for (int i = 0; i < 16; i++) L[i] = store[(int64_t)(v * 16 + i) * store_events + ev];
        }
      }
      if (phs_in(V.x_phi, seg.x_stride, PHS_CHK_ADJ)) xb[V.x_phi] = fx_mul(kr, 2.0 * PHS_PI, ph);
      if (phs_in(V.x_ct, seg.x_stride, PHS_CHK_ADJ))
        xb[V.x_ct] = ct_adjoint(kr, V.ct_class, xrow_at(xe, V.x_ct, seg.x_stride), V.b1, t.st,
                                slot(sm, ab + 4), th, ct0b, jb);
      // the rapidity is that of (E, p) at mass m: d eta = dp / E - (p / E) dmsq / (2 m^2); a
      // massless pair's own energy goes to p and msq through E^2 = p^2 + msq.  The root's are
      // constants.
      double vb_msq = 0.0, vb_p = pb_v;
      if (!V.self_root) {
        const double re = fx_rcp(E_v, kr);
        const double te = fx_mul(kr, et, re), ee = fx_mul(kr, Eb, re);
        vb_p = fma(ee, p_v, fx_add(kr, vb_p, te));
        vb_msq = fma(fx_mul(kr, -te, t.bg), hm, fx_scale(ee, -1));
      }
      // p_decay = sl / (2 m), E = (msq +- (c0 - c1)) / (2 m), log sl - log msq, with
      // dlambda = 2 (msq - c0 - c1) dmsq - 4 m (E1 dc0 + E0 dc1)
      double cmsqb0 = 0.0, cmsqb1 = 0.0;
      if (massless == 3) {
        // p_decay = E0 = E1 = m / 2, and sl / msq is 1
        vb_msq = fma(fx_scale(fx_add(kr, pcb, fx_add(kr, ceb0, ceb1)), -1), hm, vb_msq);
      } else {
        const double rs = fx_rcp(sl, kr);
        const double ldab = fx_scale(fx_mul(kr, fma(pcb, hm, fx_mul(kr, jb, rs)), rs), -1);
        const double d = fx_sub(kr, fx_sub(kr, msq_v, cmsq[0]), cmsq[1]);
        const double half = fx_scale(fma(pcb, pc, fma(ceb0, ce0, fx_mul(kr, ceb1, ce1))), -1);
        vb_msq = fma(fx_scale(ldab, 1), d, vb_msq);
        vb_msq = fma(fx_add(kr, ceb0, ceb1), hm, vb_msq);
        vb_msq = fma(fx_mul(kr, -rm, rm), fx_add(kr, half, jb), vb_msq);
        const double l4 = fx_scale(fx_mul(kr, -ldab, m_v), 2), dh = fx_mul(kr, fx_sub(kr, ceb0, ceb1), hm);
        cmsqb0 = fma(l4, ce1, dh);
        cmsqb1 = fma(l4, ce0, -dh);
      }
      // internal daughters: their msq is complete now; map it to x and the mapping parameters
#pragma unroll 1
      for (int j = 0; j < 2; j++) {
        const PhsChild &C = V.child[j];
        if (!C.internal || !phs_in(A.child_visit[j], n_visits, PHS_CHK_VISITS) ||
            !phs_in(C.x_msq, seg.x_stride, PHS_CHK_ADJ))
          continue;
        const double msqb = fx_add(kr, j == 0 ? cmsqb0 : cmsqb1, j == 0 ? c_msqb[0] : c_msqb[1]);
        double xmb, mb, wb;
        map_adjoint(kr, C, A.child[j], xrow_at(xe, C.x_msq, seg.x_stride),
                    slot(sm, lay.ang0 + PHS_ADJ_ANG * A.child_visit[j] + 5), msqb, jb, xmb, mb, wb);
        xb[C.x_msq] = xmb;
        if (2 * C.x_msq + 1 < th_stride) {
          tb[2 * C.x_msq] = mb;
          tb[2 * C.x_msq + 1] = wb;
        }
      }
      // on to the previous visit
      if (v > 0) {
        if (A.entered_by_pop && phs_in(asp, lay.depth, PHS_CHK_STACK) &&
            phs_in(A.pop_slot, lay.npops, PHS_CHK_STACK)) {
          const int base = lay.stack0 + PHS_ADJ_FRAME * asp;
#pragma unroll
          for (int i = 0; i < 16; i++) slot(sm, base + i) = Lb[i];
          slot(sm, base + 16) = vb_msq;
          slot(sm, base + 17) = vb_p;
          asp++;
#pragma unroll
          for (int i = 0; i < 16; i++) {
            L[i] = slot(sm, lay.pop0 + 16 * A.pop_slot + i);
            Lb[i] = 0.0;
          }
          sb_msq = sb_p = 0.0;
        } else {
          sb_msq = vb_msq;
          sb_p = vb_p;
        }
      }
    }
  }
}

}  // namespace

void phs_adjoint_sizes(int max_visits, int max_pops, int stack_depth, bool friends, int *state0,
                       int *ang0, int *pop0, int *stack0, int *fr0, size_t *smem) {
  *state0 = 0;
  *ang0 = PHS_ADJ_STATE * max_visits;
  *pop0 = *ang0 + PHS_ADJ_ANG * max_visits;
  *stack0 = *pop0 + 16 * max_pops;
  static_assert(PHS_ADJ_FRAME <= PHS_STATE, "the adjoint stack takes the frame stack's slots");
  *fr0 = *stack0 + PHS_STATE * (stack_depth > 0 ? stack_depth : 0);
  const int slots = *fr0 + (friends ? 3 * max_visits : 0);
  *smem = (size_t)slots * PHS_ADJ_BLOCK * sizeof(double);
}

template <bool FRIENDS, bool STORED>
static const void *adjoint_kernel() {
  return (const void *)phs_adjoint_kernel<FRIENDS, STORED>;
}

static const void *adjoint_kernel(bool friends, bool stored) {
  if (stored) return friends ? adjoint_kernel<true, true>() : adjoint_kernel<false, true>();
  return friends ? adjoint_kernel<true, false>() : adjoint_kernel<false, false>();
}

cudaError_t phs_launch_adjoint(const PhsLaunch &a, const PhsAdjChannel *adj, const double *pbar,
                               const double *jbar, double *xbar, double *thbar, int th_stride,
                               int max_visits, int max_pops, bool friends, int n_blocks,
                               cudaStream_t stream, double *store, int64_t store_events) {
  if (a.n_tiles <= 0) return cudaSuccess;
  AdjLayout lay;
  size_t smem;
  phs_adjoint_sizes(max_visits, max_pops, a.stack_depth, friends, &lay.state0, &lay.ang0, &lay.pop0,
                    &lay.stack0, &lay.fr0, &smem);
  lay.nv = max_visits;
  lay.npops = max_pops;
  lay.depth = a.stack_depth;
  const bool stored = store != nullptr;
  const void *k = adjoint_kernel(friends, stored);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
#define PHS_ADJ_LAUNCH(F, S)                                                                   \
  phs_adjoint_kernel<F, S><<<n_blocks, PHS_ADJ_BLOCK, smem, stream>>>(a, adj, pbar, jbar, xbar, \
                                                                     thbar, th_stride, lay,     \
                                                                     store, store_events)
  if (stored) {
    if (friends) PHS_ADJ_LAUNCH(true, true); else PHS_ADJ_LAUNCH(false, true);
  } else {
    if (friends) PHS_ADJ_LAUNCH(true, false); else PHS_ADJ_LAUNCH(false, false);
  }
#undef PHS_ADJ_LAUNCH
  return cudaGetLastError();
}

int phs_adjoint_blocks_per_sm(int max_visits, int max_pops, int stack_depth, bool friends,
                              bool stored) {
  int s0, a0, p0, k0, f0;
  size_t smem;
  phs_adjoint_sizes(max_visits, max_pops, stack_depth, friends, &s0, &a0, &p0, &k0, &f0, &smem);
  const void *k = adjoint_kernel(friends, stored);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, PHS_ADJ_BLOCK, smem);
  return n > 0 ? n : 1;
}

PHS_CHECK_COLLECTOR(phs_check_collect_adjoint)
