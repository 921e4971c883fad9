// phs_inverse.cu -- the inverse map: momenta of generated events -> x and factor of every
// channel (the reference's do_inverse_mapping pass of gen_phs_from_x_gpu, phs.cu:1499-1554,
// with _combine_particles 1262-1283, _apply_msq_inv 626-675, the boost inversion 924-1244
// and the inverse mappings of mappings_gpu.hpp:15-219).
//
// The reference runs this as a host loop over channels, each iteration a chain of
// event-parallel kernels (combine, msq, one launch per boost level, with and without
// friends) that round-trip msq, p_decay, phi/ct/st and a 4x4 matrix per boost through HBM.
// Here one kernel does all of it: a block takes a tile of events and the channels of one tree
// shape, lists the ok events, and each thread walks the shape's visit program (phs_program.h)
// for one of them, with the running frame in registers and the branch momenta in its
// shared-memory column; then the mappings of each channel of the shape.  Per (event, channel)
// the only HBM traffic is the x row and the factor written.
//
// The FP64 pipe bounds it, so square roots, reciprocals, angles, arctangents and logarithms
// come from phs_fix.h, the separately rounded products and sums are FMAs with register
// constants (the same bits), and what is rare is called rather than inlined: four warps of a
// block walk the same program, but different blocks do not, and with twice the code the
// instruction fetches took a sixth of the time.  2e5 events of 16 channels (6 particles):
// 6.09 -> 2.47 ms (before tiles were spread over the call 2.60; 3.45 with 64-thread blocks and the
// rare code inlined, 4.0 with 32-thread blocks).
//
// At a visit of branch b, with Gp and (theta, phi) the frame and angles of b's parent:
//   G   = [R_f^-1] B_z(-bg_b) R_y(-theta) R_z(-phi) Gp   b's rest frame, z along its flight
//                                                         (or friend) axis
//   msq of both daughters from their summed momenta; inverse msq maps of internal ones
//   Kallen function at b -> daughters' decay momentum; factor *= sqrt(lambda)/msq_b
//   q   = G p(daughter 1) -> phi = atan2(q_y, q_x), cos(theta) = q_z/|q| -> x, inverse ct map
//   (G, theta, phi) handed to the internal daughters (carry / stack)
// The friend rotation R_f is the exact rotation onto the friend beam's direction; the
// reference's differs from it only away from the root's daughters (phs.cu:1183-1244).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "phs_device.h"
#include "phs_event_f64.cuh"
#include "phs_program.h"

#define PHS_INV_STATE 23  // doubles per saved frame: G[16], ct, st, cos phi, sin phi, msq, p_decay, m
// per visit, from the geometry walk to the mapping pass: msq of both daughters, cos(theta)
// and x_phi of daughter 1, sqrt(lambda) / msq of the visited branch
#define PHS_INV_GEO 5
// per visit, the last mapping results (x, f) of daughter 0, daughter 1 and cos(theta), which
// the next channel of the shape reuses where its mapping is the same (left out when the
// block's shared memory would not hold it: the largest trees)
#define PHS_INV_CACHE 6

namespace {

// (x, f) of the STEP maps: a call, for the code's size (as map_msq_step).
__device__ __noinline__ double2 map_msq_step_inverse(int t, double msq, double s, double msq_min,
                                                     double msq_max, double a0, double a1, double a2) {
  const double z1 = (msq - msq_min) / (msq_max - msq_min);
  if (t == PHS_MAP_STEP_E) {
    const double z2 = 1.0 + a1 * exp(z1 / a2);
    return make_double2((z1 - a2 * log(z2 / (1.0 + a1))) / a0, a0 * z2 * (msq_max - msq_min) / s);
  }
  const double z3 = a0 - z1 / a2;
  const double x = ((a0 + z1 / a2 + z1) - sqrt(z3 * z3 + 2.0 * z1 * (a0 + z1 / a2) + z1 * z1)) / 2.0;
  return make_double2(x, (a1 / (a0 - x) / (a0 - x) + a2) * (msq_max - msq_min) / s);
}

// mappings_gpu.hpp:15-172 (mapping_x_from_msq_*), constants as in phs_cpu.cpp:452-531.
__device__ __forceinline__ void map_msq_inverse(const FxRegs &k, int t, double msq, double s,
                                                double m, double w, double msq_min,
                                                double msq_max, double a0, double a1, double a2,
                                                double &x, double &f) {
  switch (t) {
    case PHS_MAP_NO:
      x = fx_div(fx_sub(k, msq, msq_min), fx_sub(k, msq_max, msq_min), k);
      f = a2;
      break;
    case PHS_MAP_COLLINEAR:
    case PHS_MAP_INFRARED:
    case PHS_MAP_RADIATION: {
      const double z = fx_add(k, fx_sub(k, msq, msq_min), a0);
      x = fx_div(fx_log(fx_div(z, a0, k)), a1, k);
      f = fx_mul(k, a2, z);
      break;
    }
    case PHS_MAP_TCHANNEL:
    case PHS_MAP_UCHANNEL: {
      // one logarithm per lane: the side of the midpoint selects its argument
      const bool lower = fx_gt(fx_scale(fx_add(k, msq_max, msq_min), -1), msq);
      const double z = fx_add(k, lower ? fx_sub(k, msq, msq_min) : fx_sub(k, msq_max, msq), a0);
      const double lx = fx_div(fx_log(fx_div(z, a0, k)), a1, k);
      x = lower ? lx : fx_sub(k, k.one, lx);
      f = fx_mul(k, a2, z);
      break;
    }
    case PHS_MAP_STEP_E:
    case PHS_MAP_STEP_H: {
      const double2 r = map_msq_step_inverse(t, msq, s, msq_min, msq_max, a0, a1, a2);
      x = r.x;
      f = r.y;
      break;
    }
    default:
      x = 0.0;
      f = 0.0;
  }
}

// mappings_gpu.hpp:184-219 (mapping_x_from_ct_*).
__device__ __forceinline__ void map_ct_inverse(const FxRegs &k, int ct_class, double ct, double b0,
                                               double b1, double &x, double &f) {
  if (ct_class == PHS_CT_COLLINEAR) {
    // one logarithm per lane, as for the msq maps
    const bool lower = ct < 0.0;
    const double ct1 = fx_add(k, fx_add(k, lower ? ct : fx_neg(ct), b0), k.one);
    const double lx = fx_div(fx_log(fx_div(ct1, b0, k)), fx_scale(b1, 1), k);
    x = lower ? lx : fx_sub(k, k.one, lx);
    f = fx_mul(k, ct1, b1);
  } else {
    x = fx_scale(fx_add(k, ct, k.one), -1);
    f = 1.0;
  }
}

__device__ __forceinline__ void inv_store(double *stk, int depth, int k, double v) {
  stk[(depth * PHS_INV_STATE + k) * PHS_INV_BLOCK + threadIdx.x] = v;
}
__device__ __forceinline__ double inv_load(const double *stk, int depth, int k) {
  return stk[(depth * PHS_INV_STATE + k) * PHS_INV_BLOCK + threadIdx.x];
}

// Momentum slots of one thread's event: slot j < n_out is outgoing particle j, slot
// n_out + i the i-th internal branch in post-order.  Internal sums sit in shared memory at
// pm[(4 (j - n_out) + mu) PHS_INV_BLOCK].  The outgoing momenta are either staged in shared
// memory below them (pm[(4 j + mu) PHS_INV_BLOCK], the CM momenta after the inverse lab
// boost) or, where there is no lab boost (CM = lab, the same bits), read from the event's
// row of p through the L1 (lab != null): that leaves 4 n_out doubles per thread of shared
// memory free for more resident blocks.
struct InvMomenta {
  double *pm;          // internal sums (and, lab == null, the staged outgoing momenta first)
  const double *lab;   // the event's p row, or null
  int n_out;
  // checked build: slot j of the 2 n_out - 1 (the root's sum is never formed or read)
  __device__ __forceinline__ double get(int j, int mu) const {
    if (!phs_in(j, 2 * n_out - 2, PHS_CHK_SLOT)) return 0.0;
    if (lab) return j < n_out ? __ldg(lab + 4 * j + mu) : pm[(4 * (j - n_out) + mu) * PHS_INV_BLOCK];
    return pm[(4 * j + mu) * PHS_INV_BLOCK];
  }
  __device__ __forceinline__ void set_internal(int j, int mu, double v) const {
    if (!phs_in(j - n_out, n_out - 2, PHS_CHK_SLOT)) return;
    pm[(4 * (lab ? j - n_out : j) + mu) * PHS_INV_BLOCK] = v;
  }
};

// The geometry of one (event, channel shape): the walk of the visit program without the
// mappings, leaving per visit in geo (slot (v PHS_INV_GEO + k) PHS_INV_BLOCK) what the
// mappings of every channel of that shape need (inverse_maps).
// The arithmetic keeps the reference's operation order (this file is compiled without
// contraction): x(p) is ill-conditioned near the poles of each decay (cos(theta) -> +-1,
// where 1 - cos^2 cancels) and for soft daughters of fast branches, and there any other
// rounding order moves the result by far more than the input's own rounding does.  The
// exceptions are divisions by constants of an output that is not ill-conditioned in them,
// done as products with the constant's reciprocal (one rounding more): x_phi = phi / 2 pi
// and the Breit-Wigner inverse's divisions by m w and a1 - a0.
__device__ void inverse_geometry(const FxRegs &k, const PhsChannel &ch, const InvMomenta &pm, double sqrts,
                                 double *stk, double *geo, int stack_depth) {
  const double s = fx_mul(k, sqrts, sqrts);
  const auto mul = [&](double u, double v) { return fx_mul(k, u, v); };
  const auto add = [&](double u, double v) { return fx_add(k, u, v); };
  const auto sub = [&](double u, double v) { return fx_sub(k, u, v); };
  // internal momenta as sums of their daughters in post-order (_combine_particles,
  // phs.cu:1262-1283); the root's (the last) is never a daughter
  for (int i = 0; i + 1 < ch.n_vol; i++) {
    const int a = ch.comb[i][0], b = ch.comb[i][1], o = ch.n_out + i;
#pragma unroll
    for (int mu = 0; mu < 4; mu++) pm.set_internal(o, mu, add(pm.get(a, mu), pm.get(b, mu)));
  }
  // carried state of the visited branch: its parent's frame Gp and angles, its msq, decay
  // momentum and mass
  double Gp[16];
  double ct0 = 1.0, st0 = 0.0, cp0 = 1.0, sp0 = 0.0;
  double msq_b = s, pd_b = 0.0, m_b = sqrts;
  int sp = 0;
  const int n_visits = ch.n_visits;
  for (int v = 0; v < n_visits; v++) {
    const PhsVisit &V = ch.visit[v];
    // one reciprocal of the mass serves both divisions by it
    const bool serves = fx_quot_serves(m_b);
    const double rm = serves ? fx_rcp(m_b, k) : 0.0;
    // the branch's frame G: CM momenta -> its rest frame, z along its flight (or friend)
    // axis.  The root's is the identity; else L_r3_r2_b3(-bg, gamma, ct0, -st0, cp0, -sp0)
    // times the parent's (phs.cu:1114-1125)
    double G[16];
    if (V.self_root) {
#pragma unroll
      for (int i = 0; i < 16; i++) G[i] = (i % 5 == 0) ? 1.0 : 0.0;
    } else {
      const double bg = fx_gt(m_b, 0.0) ? (serves ? fx_quot(pd_b, m_b, rm, k) : fx_lib_div(pd_b, m_b)) : 0.0;
      const double ga = fx_sqrt(add(mul(bg, bg), k.one), k);
      const double bs = mul(-bg, st0), gs = mul(ga, st0);
      const double t01 = mul(bs, cp0), t02 = mul(bs, sp0), t03 = mul(-bg, ct0);
      const double t11 = mul(ct0, cp0), t12 = mul(ct0, sp0);
      const double t31 = mul(gs, cp0), t32 = mul(gs, sp0), t33 = mul(ga, ct0);
      if (V.parent_root) {
        // the parent's frame is the root's, the identity: G is the step's own matrix (the
        // product below with Gp = 1 gives the same bits)
        G[0] = ga;    G[1] = t01;   G[2] = t02;  G[3] = t03;
        G[4] = 0.0;   G[5] = t11;   G[6] = t12;  G[7] = fx_neg(st0);
        G[8] = 0.0;   G[9] = fx_neg(sp0); G[10] = cp0; G[11] = 0.0;
        G[12] = fx_neg(bg); G[13] = t31;  G[14] = t32; G[15] = t33;
      } else {
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const double g0 = Gp[c], g1 = Gp[4 + c], g2 = Gp[8 + c], g3 = Gp[12 + c];
          // row 0 only feeds the frames of internal daughters
          G[c] = g0;   // row 0 below
          G[4 + c] = add(add(mul(t11, g1), mul(t12, g2)), mul(-st0, g3));
          G[8 + c] = add(mul(-sp0, g1), mul(cp0, g2));
          G[12 + c] = add(add(add(mul(-bg, g0), mul(t31, g1)), mul(t32, g2)), mul(t33, g3));
        }
        // row 0 only feeds the frames of internal daughters (a loop: the compiler would issue
        // a short block's FP64 instructions also where it is skipped)
#pragma unroll 1
        for (int c = V.both_leaves ? 4 : 0; c < 4; c += 4) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            G[i] = add(add(add(mul(ga, Gp[i]), mul(t01, Gp[4 + i])), mul(t02, Gp[8 + i])), mul(t03, Gp[12 + i]));
        }
      }
      if (V.friend_sign != 0) {
        // rotate the friend beam's direction G (1, 0, 0, ff) onto z (phs.cu:1183-1206);
        // uniform per channel
        const double ff = V.friend_sign;
        double Rf[9];
        rot_z_onto(G[4] + ff * G[7], G[8] + ff * G[11], G[12] + ff * G[15], Rf);
        double Gn[12];
#pragma unroll
        for (int r = 0; r < 3; r++)
#pragma unroll
          for (int c = 0; c < 4; c++)
            Gn[4 * r + c] = Rf[r] * G[4 + c] + Rf[3 + r] * G[8 + c] + Rf[6 + r] * G[12 + c];
#pragma unroll
        for (int i = 0; i < 12; i++) G[4 + i] = Gn[i];
      }
    }

    // daughters' momenta and invariant masses
    double q0[4], q1[4];
#pragma unroll
    for (int mu = 0; mu < 4; mu++) {
      q0[mu] = pm.get(V.slot[0], mu);
      q1[mu] = pm.get(V.slot[1], mu);
    }
    double cmsq[2];
    cmsq[0] = sub(sub(sub(mul(q0[0], q0[0]), mul(q0[1], q0[1])), mul(q0[2], q0[2])), mul(q0[3], q0[3]));
    cmsq[1] = sub(sub(sub(mul(q1[0], q1[0]), mul(q1[1], q1[1])), mul(q1[2], q1[2])), mul(q1[3], q1[3]));

    geo[(PHS_INV_GEO * v + 0) * PHS_INV_BLOCK] = cmsq[0];
    geo[(PHS_INV_GEO * v + 1) * PHS_INV_BLOCK] = cmsq[1];

    // Kallen function at the visited branch
    const double d = sub(sub(msq_b, cmsq[0]), cmsq[1]);
    const double sl = fx_sqrt(sub(mul(d, d), mul(fx_scale(cmsq[0], 2), cmsq[1])), k);
    // (halving sl / m and dividing by 2 m round alike)
    const double pd = serves ? fx_scale(fx_quot(sl, m_b, rm, k), -1) : fx_lib_div(sl, 2.0 * m_b);
    geo[(PHS_INV_GEO * v + 4) * PHS_INV_BLOCK] = fx_div(sl, msq_b, k);

    // angles of daughter 1 in the branch's frame (azimuthal_angle, polar_angle_ct,
    // phs.cu:913-922)
    // (the root's frame is the identity: the same bits without the products)
    double qx = q0[1], qy = q0[2], qz = q0[3];
#pragma unroll 1
    for (int r = V.self_root ? 1 : 0; r < 1; r++) {
      qx = add(add(add(mul(G[4], q0[0]), mul(G[5], q0[1])), mul(G[6], q0[2])), mul(G[7], q0[3]));
      qy = add(add(add(mul(G[8], q0[0]), mul(G[9], q0[1])), mul(G[10], q0[2])), mul(G[11], q0[3]));
      qz = add(add(add(mul(G[12], q0[0]), mul(G[13], q0[1])), mul(G[14], q0[2])), mul(G[15], q0[3]));
    }
    double phi = fx_atan2(qy, qx);
    if (fx_bits(phi) > 0x8000000000000000ull) phi = add(phi, 2.0 * PHS_PI);   // below 0 (-0 is not)
    geo[(PHS_INV_GEO * v + 3) * PHS_INV_BLOCK] = mul(phi, 1.0 / (2.0 * PHS_PI));   // x_phi
    const double ct = fx_div(qz, fx_sqrt(add(add(mul(qx, qx), mul(qy, qy)), mul(qz, qz)), k), k);
    geo[(PHS_INV_GEO * v + 2) * PHS_INV_BLOCK] = ct;
    if (V.both_leaves) {
      if (sp > 0) {
        sp--;
#pragma unroll
        for (int i = 0; i < 16; i++) Gp[i] = inv_load(stk, sp, i);
        ct0 = inv_load(stk, sp, 16);
        st0 = inv_load(stk, sp, 17);
        cp0 = inv_load(stk, sp, 18);
        sp0 = inv_load(stk, sp, 19);
        msq_b = inv_load(stk, sp, 20);
        pd_b = inv_load(stk, sp, 21);
        m_b = inv_load(stk, sp, 22);
      }
      continue;
    }
    const double st = fx_sqrt(sub(k.one, mul(ct, ct)), k);
    double sph, cph;
    fx_sincos(phi, sph, cph);
    if (V.push >= 0 && phs_in(sp, stack_depth, PHS_CHK_STACK)) {
      const bool j0 = V.push == 0;
#pragma unroll
      for (int i = 0; i < 16; i++) inv_store(stk, sp, i, G[i]);
      inv_store(stk, sp, 16, ct);
      inv_store(stk, sp, 17, st);
      inv_store(stk, sp, 18, cph);
      inv_store(stk, sp, 19, sph);
      const double mq = j0 ? cmsq[0] : cmsq[1];
      inv_store(stk, sp, 20, mq);
      inv_store(stk, sp, 21, j0 ? pd : fx_neg(pd));
      inv_store(stk, sp, 22, fx_sqrt(mq, k));
      sp++;
    }
    if (V.carry >= 0) {
      const bool j0 = V.carry == 0;
#pragma unroll
      for (int i = 0; i < 16; i++) Gp[i] = G[i];
      ct0 = ct;
      st0 = st;
      cp0 = cph;
      sp0 = sph;
      msq_b = j0 ? cmsq[0] : cmsq[1];
      pd_b = j0 ? pd : fx_neg(pd);
      m_b = fx_sqrt(msq_b, k);
    }
  }
}

// The mappings of one (event, channel) after inverse_geometry of its shape: writes the
// channel's x entries of xr and returns its factor, in the reference's order of factors.
// Bit 3 v + k of reuse (k = 0, 1: the daughters' msq maps, 2: the cos(theta) map): the
// previous channel of the shape had the same mapping there, so its (x, f) is taken from
// cache (null: no cache, reuse 0).  xr null: the mappings run (the next channel may reuse
// them) but write nothing.
template <bool PER_EVENT>
__device__ double inverse_maps(const FxRegs &k, const PhsChannel &ch, double sqrts, const double *geo,
                               double *cache, double *xr, uint64_t reuse, int n_x) {
  const double s = fx_mul(k, sqrts, sqrts);
  double factor = 1.0;
  const int n_visits = ch.n_visits;
  for (int v = 0; v < n_visits; v++) {
    const PhsVisit &V = ch.visit[v];
    // inverse msq maps of the internal daughters (not unrolled: the code of one serves both)
#pragma unroll 1
    for (int j = 0; j < 2; j++) {
      const PhsChild &C = V.child[j];
      if (C.internal) {
        double *slot = cache ? cache + (PHS_INV_CACHE * v + 2 * j) * PHS_INV_BLOCK : nullptr;
        double x, f;
        if (reuse >> (3 * v + j) & 1) {
          x = slot[0];
          f = slot[PHS_INV_BLOCK];
        } else {
          double a0 = C.a0, a1 = C.a1, a2 = C.a2, mn = C.msq_min, mx = C.msq_max, mmax;
          if (PER_EVENT) child_constants(k, C, sqrts, ch.m_tot, fx_rcp(s, k), a0, a1, a2, mn, mx, mmax);
          const double msq = geo[(PHS_INV_GEO * v + j) * PHS_INV_BLOCK];
          if (C.map_id == PHS_MAP_SCHANNEL) {
            // mapping_x_from_msq_schannel with its divisors m w and a1 - a0 (constants of the
            // channel) as compiled reciprocals
            const double z = fx_mul(k, fx_sub(k, msq, C.msq0), C.inv_mw);
            const double da = fx_sub(k, fx_atan2(z, 1.0), a0);
            x = PER_EVENT ? fx_div(da, fx_sub(k, a1, a0), k) : fx_mul(k, da, C.inv_da);
            f = fx_mul(k, a2, fx_add(k, fx_mul(k, z, z), k.one));
          } else {
            map_msq_inverse(k, C.map_id, msq, s, C.m, C.w, mn, mx, a0, a1, a2, x, f);
          }
          if (slot) {
            slot[0] = x;
            slot[PHS_INV_BLOCK] = f;
          }
        }
        if (xr && phs_in(C.x_msq, n_x, PHS_CHK_INV)) xr[C.x_msq] = x;
        factor = fx_mul(k, factor, f);
      }
    }
    factor = fx_mul(k, factor, geo[(PHS_INV_GEO * v + 4) * PHS_INV_BLOCK]);  // sqrt(lambda) / msq
    if (xr && phs_in(V.x_phi, n_x, PHS_CHK_INV)) xr[V.x_phi] = geo[(PHS_INV_GEO * v + 3) * PHS_INV_BLOCK];
    double *slot = cache ? cache + (PHS_INV_CACHE * v + 4) * PHS_INV_BLOCK : nullptr;
    double x, f;
    if (reuse >> (3 * v + 2) & 1) {
      x = slot[0];
      f = slot[PHS_INV_BLOCK];
    } else {
      double b0 = V.b0, b1 = V.b1;
      if (PER_EVENT && V.ct_class == PHS_CT_COLLINEAR) {
        b0 = V.m * V.m / s;
        b1 = log((b0 + 1.0) / b0);
      }
      map_ct_inverse(k, V.ct_class, geo[(PHS_INV_GEO * v + 2) * PHS_INV_BLOCK], b0, b1, x, f);
      if (slot) {
        slot[0] = x;
        slot[PHS_INV_BLOCK] = f;
      }
    }
    if (xr && phs_in(V.x_ct, n_x, PHS_CHK_INV)) xr[V.x_ct] = x;
    if (V.ct_class == PHS_CT_COLLINEAR) factor = fx_mul(k, factor, f);   // uniform: 1
  }
  return factor;
}

// The block's shared memory beside the dynamic one (phs_inverse_smem_bytes).
struct InvShared {
  uint16_t listed[PHS_INV_TILE];  // the tile's ok events
  int warp_ok[PHS_INV_BLOCK / 32], next_work;
};

// One block: `tile` events and the channels of one tree shape (in the launch's slice of the
// group order).  It gathers the tile's ok events and walks them, a warp 32 at a time, and writes
// the outputs that need no arithmetic.  What bounds the kernel is the FP64 pipe; events are ok in
// very different shares from channel to channel, so a tile is chunks of PHS_INV_CHUNK events spread
// evenly over all of them, and blocks differ little.  (Contiguous tiles: 2e5 events of 16 channels 2.60
// ms, 2.47 so; 2e5 of 16 channels of 8 particles 1.26 -> 1.04.  Persistent blocks that each took 64
// events through every channel left most SMs idle: 40 000 ok events of 2e5 are 600 such walks.)
// The other outputs are written beside the walks: ahead of them, with one block on an SM, 2e5
// events of 8 channels of 12 particles, 12 % of them ok, took 1.08 ms instead of 0.92.
// LAB_ROWS: no lab boost (uniform beams with E1 = E2): the outgoing momenta are read from p
// instead of staged in shared memory (InvMomenta).
template <bool PER_EVENT, bool LAB_ROWS>
__global__ void __launch_bounds__(PHS_INV_BLOCK, 3)
    phs_inverse_kernel(const __grid_constant__ PhsInvLaunch a) {
  static_assert(!(PER_EVENT && LAB_ROWS), "per-event beams stage their CM momenta");
  constexpr int kWarps = PHS_INV_BLOCK / 32, kChunk = PHS_INV_CHUNK;
  extern __shared__ double sm[];
  const FxRegs k = fx_regs();
  double *pm = sm;  // [4 (n_out - 1), or 4 (2 n_out - 1) with staging][block]
  double *stk = sm + (size_t)4 * (LAB_ROWS ? a.n_out - 1 : 2 * a.n_out - 1) * PHS_INV_BLOCK;  // frame stack
  double *geo = stk + (size_t)PHS_INV_STATE * a.stack_depth * PHS_INV_BLOCK;  // per-visit geometry
  double *cache = a.group_reuse ? geo + (size_t)PHS_INV_GEO * a.max_visits * PHS_INV_BLOCK
                                : nullptr;  // per-visit mapping results
  __shared__ InvShared sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n_groups = a.group_hi - a.group_lo;
  const int64_t per_group = (a.n_events + a.tile - 1) / a.tile, n_items = per_group * n_groups;
  const int64_t n_chunks = (a.n_events + kChunk - 1) / kChunk;
  const bool has_own = a.x_own != nullptr;

  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int g = a.group_lo + (int)(item % n_groups);
    // the block's chunks: first, first + per_group, ..  (entry j: chunk j / kChunk of them)
    const int64_t first = item / n_groups;
    const int n_ch = (int)((n_chunks - first + per_group - 1) / per_group);
    const auto event = [&](int j) { return ((int64_t)(j / kChunk) * per_group + first) * kChunk + j % kChunk; };
    const int gb = a.group_begin[g], ge = a.group_begin[g + 1];
    const int lo = max(gb, a.order_lo), hi = min(ge, a.order_hi);
    // checked build: the group's entries, its shape's program, the regions sized for it and
    // the tile (block-uniform: every thread leaves together)
    if (!phs_in(gb, a.n_channels, PHS_CHK_SLOT) || !phs_in(hi - 1, a.n_channels, PHS_CHK_SLOT) ||
        !phs_in(a.group_order[gb], a.n_channels, PHS_CHK_CHANNEL) ||
        !phs_in(a.channels[a.group_order[gb]].n_visits - 1, a.max_visits, PHS_CHK_VISITS) ||
        !phs_in(a.channels[a.group_order[gb]].n_out - 1, a.n_out, PHS_CHK_SLOT) ||
        !phs_in(n_ch * kChunk - 1, PHS_INV_TILE, PHS_CHK_SLOT) ||
        !phs_in(min(event(n_ch * kChunk - 1), a.n_events - 1), a.x_ch_stride, PHS_CHK_INV))
      continue;

    // 1. the ok events, listed in order: the inversions run in full warps (an FP64 instruction
    // costs the pipe the same whatever the number of active lanes).  A shape's only channel
    // does not invert the events that it generated.
    const bool skip_own = has_own && hi - lo == 1;
    const int c0 = a.group_order[lo];
    const int64_t skip0 = skip_own ? a.ch_begin[c0] : 0;
    const int64_t skip1 = skip_own ? (c0 + 1 < a.n_channels ? a.ch_begin[c0 + 1] : a.n_events) : 0;
    int n_list = 0;  // block-uniform
    if (tid == 0) sh.next_work = 0;   // (read after the barriers below)
    for (int base = 0; base < n_ch * kChunk; base += PHS_INV_BLOCK) {
      const int j = base + tid;
      const int64_t e = event(j);
      const bool take = j < n_ch * kChunk && e < a.n_events && (!a.ok || a.ok[e]) && !(e >= skip0 && e < skip1);
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (lane == 0) sh.warp_ok[wid] = __popc(m);
      __syncthreads();
      int before = n_list, total = 0;
      for (int w = 0; w < kWarps; w++) {
        if (w < wid) before += sh.warp_ok[w];
        total += sh.warp_ok[w];
      }
      const int d = before + __popc(m & ((1u << lane) - 1u));
      if (take && phs_in(d, PHS_INV_TILE, PHS_CHK_SLOT)) sh.listed[d] = (uint16_t)j;
      n_list += total;
      __syncthreads();  // warp_ok is read, the entries are written
    }

    // 2. the warps take what there is to do from a counter: first walks of 32 listed events (the
    // geometry once per event, then the mappings of each channel of the shape), then pieces of the
    // outputs that need no arithmetic, so that warps without a walk write beside those with one
    const int n_walks = (n_list + 31) / 32, n_work = n_walks + n_ch * (hi - lo);
    for (;;) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&sh.next_work, 1);
      at = __shfl_sync(0xffffffffu, at, 0);
      if (at >= n_work) break;
      if (at >= n_walks) {
        // per channel the generating channel's own x and factor, x padding beyond a channel's
        // n_x_used, zeros for ok = false events; rows of consecutive events are contiguous
        const int i = lo + (at - n_walks) / n_ch;
        const int c = a.group_order[i];
        if (!phs_in(c, a.n_channels, PHS_CHK_CHANNEL)) continue;
        const int64_t ep = event((at - n_walks) % n_ch * kChunk);
        const int n_p = (int)min((int64_t)kChunk, a.n_events - ep);
        const int64_t own0 = a.ch_begin[c] - ep;
        const int64_t own1 = (c + 1 < a.n_channels ? a.ch_begin[c + 1] : a.n_events) - ep;
        const int n_used = a.channels[c].n_x_used;
        double *xr = a.x_out + ((int64_t)c * a.x_ch_stride + ep) * a.n_x;
        const double *xo = has_own ? a.x_own + ep * a.n_x : nullptr;
        int ev = lane / a.n_x, kx = lane - ev * a.n_x;
        const int dev = 32 / a.n_x, dkx = 32 - dev * a.n_x;
        for (int j = lane; j < n_p * a.n_x; j += 32) {
          const bool own = has_own && ev >= own0 && ev < own1;
          if (own || kx >= n_used)
            xr[j] = xo ? xo[j] : 0.0;
          else if (a.ok && !a.ok[ep + ev])
            xr[j] = 0.0;
          ev += dev;
          kx += dkx;
          if (kx >= a.n_x) {
            kx -= a.n_x;
            ev++;
          }
        }
        for (int j = lane; j < n_p; j += 32) {
          double *fo = a.all_factors + (ep + j) * a.n_channels + c;
          if (has_own && j >= own0 && j < own1)
            *fo = a.factor_own ? a.factor_own[ep + j] : 0.0;
          else if (a.ok && !a.ok[ep + j])
            *fo = 0.0;
        }
        continue;
      }
      const int slot = at * 32 + lane;
      if (slot < n_list && phs_in(event(sh.listed[slot]), a.n_events, PHS_CHK_SLOT)) {
        const int64_t e = event(sh.listed[slot]);
        const PhsChannel &ch0 = a.channels[0];
        double sqrts = ch0.sqrts, lab_bg = ch0.lab ? ch0.lab_bg : 0.0;
        double lab_ga = ch0.lab ? ch0.lab_gamma : 1.0;
        if (PER_EVENT) {
          const double E1 = a.E1[e], E2 = a.E2[e], r = fx_sqrt(fx_mul(k, E1, E2), k);
          sqrts = fx_add(k, r, r);
          lab_bg = fx_div(fx_sub(k, E1, E2), sqrts, k);
          lab_ga = fx_sqrt(fx_add(k, fx_mul(k, lab_bg, lab_bg), k.one), k);
        }
        // this event's momenta, lab -> CM (the inverse of phs.cu:1286-1301)
        const double *prow = a.p + e * 4 * (int64_t)a.n_out;
        if (!LAB_ROWS) {
          const double2 *pe = reinterpret_cast<const double2 *>(prow);
          for (int q = 0; q < a.n_out; q++) {
            const double2 e_x = pe[2 * q], y_z = pe[2 * q + 1];
            pm[(4 * q + 0) * PHS_INV_BLOCK + tid] = fx_sub(k, fx_mul(k, lab_ga, e_x.x), fx_mul(k, lab_bg, y_z.y));
            pm[(4 * q + 1) * PHS_INV_BLOCK + tid] = e_x.y;
            pm[(4 * q + 2) * PHS_INV_BLOCK + tid] = y_z.x;
            pm[(4 * q + 3) * PHS_INV_BLOCK + tid] = fx_add(k, fx_mul(k, -lab_bg, e_x.x), fx_mul(k, lab_ga, y_z.y));
          }
        }
        const InvMomenta mom{pm + tid, LAB_ROWS ? prow : nullptr, a.n_out};
        inverse_geometry(k, a.channels[a.group_order[gb]], mom, sqrts, stk, geo + tid, a.stack_depth);
        for (int i = lo; i < hi; i++) {
          const int c = a.group_order[i];
          if (!phs_in(c, a.n_channels, PHS_CHK_CHANNEL) ||
              !phs_in(a.channels[c].n_visits - 1, a.max_visits, PHS_CHK_VISITS))
            continue;
          // the generating channel keeps its own row, but its mappings still run when a
          // later channel of the shape reuses them
          const bool own_row = has_own && e >= a.ch_begin[c] &&
                               (c + 1 == a.n_channels || e < a.ch_begin[c + 1]);
          if (own_row && (!cache || i + 1 == hi || a.group_reuse[i + 1] == 0)) continue;
          double *xr = own_row ? nullptr : a.x_out + ((int64_t)c * a.x_ch_stride + e) * a.n_x;
          // the first channel of a shape (or of the slice) computes every mapping
          const uint64_t reuse = i == lo || !cache ? 0ull : a.group_reuse[i];
          const double fac = inverse_maps<PER_EVENT>(k, a.channels[c], sqrts, geo + tid,
                                                     cache ? cache + tid : nullptr, xr, reuse, a.n_x);
          if (!own_row) a.all_factors[e * a.n_channels + c] = fac;
        }
      }
    }
    __syncthreads();  // the list is read, the counter was
  }
}

}  // namespace

size_t phs_inverse_smem_bytes(int n_out, int stack_depth, int max_visits, bool cache, bool lab_rows) {
  return ((size_t)4 * (lab_rows ? n_out - 1 : 2 * n_out - 1) + (size_t)PHS_INV_STATE * stack_depth +
          (size_t)(PHS_INV_GEO + (cache ? PHS_INV_CACHE : 0)) * max_visits) *
         PHS_INV_BLOCK * sizeof(double);
}

bool phs_inverse_fits_cache(int n_out, int stack_depth, int max_visits) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return phs_inverse_smem_bytes(n_out, stack_depth, max_visits, true, false) + sizeof(InvShared) <= (size_t)optin;
}

static const void *inverse_kernel(bool per_event, bool lab_rows) {
  if (per_event) return (const void *)phs_inverse_kernel<true, false>;
  return lab_rows ? (const void *)phs_inverse_kernel<false, true>
                  : (const void *)phs_inverse_kernel<false, false>;
}

int phs_inverse_blocks_per_sm(int n_out, int stack_depth, int max_visits, bool per_event,
                              bool cache, bool lab_rows) {
  int n = 0;
  lab_rows = lab_rows && !per_event;
  const size_t smem = phs_inverse_smem_bytes(n_out, stack_depth, max_visits, cache, lab_rows);
  const void *k = inverse_kernel(per_event, lab_rows);
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, PHS_INV_BLOCK, smem);
  return n > 0 ? n : 1;
}

cudaError_t phs_launch_inverse(const PhsInvLaunch &a, cudaStream_t stream) {
  if (a.n_events <= 0 || a.group_lo >= a.group_hi) return cudaSuccess;
  const bool per_event = a.E1 && a.E2;
  const bool lab_rows = !per_event && !a.lab;
  const size_t smem = phs_inverse_smem_bytes(a.n_out, a.stack_depth, a.max_visits,
                                             a.group_reuse != nullptr, lab_rows);
  const void *k = inverse_kernel(per_event, lab_rows);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int64_t n_blocks = (a.n_events + a.tile - 1) / a.tile * (a.group_hi - a.group_lo);
  const unsigned grid = (unsigned)(n_blocks < 0x7fffffff ? n_blocks : 0x7fffffff);
  if (per_event)
    phs_inverse_kernel<true, false><<<grid, PHS_INV_BLOCK, smem, stream>>>(a);
  else if (lab_rows)
    phs_inverse_kernel<false, true><<<grid, PHS_INV_BLOCK, smem, stream>>>(a);
  else
    phs_inverse_kernel<false, false><<<grid, PHS_INV_BLOCK, smem, stream>>>(a);
  return cudaGetLastError();
}

PHS_CHECK_COLLECTOR(phs_check_collect_inverse)
