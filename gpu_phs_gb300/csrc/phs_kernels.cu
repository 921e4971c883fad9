// phs_kernels.cu -- fused forward phase-space kernel (FP64) and the Philox x generator.
//
// One persistent kernel per batch.  Each warp takes 32-event tiles of one channel (tiles
// never straddle channels, so every branch of the visit program is warp-uniform); each
// thread walks its event's visit program top-down (phs_program.h) with the running 4x4
// boost in registers and at most two saved frames on a per-thread shared-memory stack.
//
// The per-event arithmetic is in phs_event_f64.cuh.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <mutex>

#include "phs_device.h"
#include "phs_event_f64.cuh"
#include "phs_program.h"

namespace {

// COMPACT: events whose kinematic test fails need no angles or boosts.  Where many fail
// (low ok fractions: multi-channel batches, hard cuts), pass A tests each event, writes
// the failures, and queues the rest per warp; pass B runs them densely.  Where nearly all
// pass, the plain loop avoids the second msq evaluation; the launcher times both.
// BLOCK threads per block (the block shape the autotuner tries), MIN_BLOCKS resident.
template <bool PER_EVENT, bool COMPACT, int MIN_BLOCKS, int BLOCK = PHS_FWD_BLOCK>
__global__ void __launch_bounds__(BLOCK, MIN_BLOCKS)
    phs_forward_f64_kernel(const __grid_constant__ PhsLaunch a) {
  extern __shared__ double smem[];
  const FxRegs k = fx_regs();
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if constexpr (COMPACT) {
    int64_t *q = reinterpret_cast<int64_t *>(smem + (size_t)a.stack_depth * PHS_STATE * BLOCK) +
                 (threadIdx.x >> 5) * 64;
    compacting_loop<0>(
        a, q,
        [&](const PhsSegment &sg, int64_t loc) { return phs_ok_f64<PER_EVENT, BLOCK>(a, k, sg, loc, smem); },
        [&](int, const PhsSegment &sg, int64_t loc) {
          if (loc >= 0) phs_event_f64<PER_EVENT, BLOCK>(a, k, sg, loc, smem);
        });
  } else {
    for (int64_t tile = warp0; tile < a.n_tiles; tile += n_warps) {
      // the segment holding this tile (warp-uniform binary search on tile_begin)
      const PhsSegment *segs = a.n_segments <= PHS_INLINE_SEGS ? a.seg_inline : a.segments;
      int lo = 0, hi = a.n_segments - 1;
      while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (segs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
      }
      const PhsSegment seg = segs[lo];
      const int64_t local = (tile - seg.tile_begin) * 32 + lane;
      if (local >= seg.ev_count) continue;
      phs_event_f64<PER_EVENT, BLOCK>(a, k, seg, local, smem);
    }
  }
}

// Split form of the FP64 kernel: after the FP32 pre-test (phs_launch_pretest, which writes
// the outputs of the events that fail for certain and queues the others per segment), the
// FP64 walk over the queued events, 32 of one segment per warp claim (a.work counts the
// claims, zeroed before the launch).  The pre-test only settles failures that the FP64
// test makes too, so the outputs are the one-pass kernel's bits.  Uniform beams only.
template <int MIN_BLOCKS, int BLOCK = PHS_FWD_BLOCK>
__global__ void __launch_bounds__(BLOCK, MIN_BLOCKS)
    phs_f64_walk_kernel(const __grid_constant__ PhsLaunch a) {
  extern __shared__ double smem[];
  const FxRegs k = fx_regs();
  const int lane = threadIdx.x & 31;
  const PhsSegment *segs = a.n_segments <= PHS_INLINE_SEGS ? a.seg_inline : a.segments;
  __shared__ int64_t tiles[PHS_INLINE_SEGS + 1];
  const int64_t *pass_tile = claim_numbering(a, tiles);
  const int64_t n_claims = pass_tile[a.n_segments];
  for (;;) {
    unsigned long long c = 0;
    if (lane == 0) c = atomicAdd(a.work, 1ull);
    const int64_t t = (int64_t)__shfl_sync(0xffffffffu, c, 0);
    if (t >= n_claims) break;
    // the last segment whose first claim is <= t (empty segments share the next one's)
    int lo = 0, hi = a.n_segments - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pass_tile[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const PhsSegment seg = segs[lo];
    const int64_t idx = (t - pass_tile[lo]) * 32 + lane;
    if (idx >= (int64_t)a.pass_count[lo]) continue;
    if (!phs_in(idx, seg.ev_count, PHS_CHK_QUEUE) ||
        !phs_in(seg.tile_begin * 32 + idx, a.n_tiles * 32, PHS_CHK_QUEUE))
      continue;
    phs_event_f64<false, BLOCK>(a, k, seg, a.pass_queue[seg.tile_begin * 32 + idx], smem);
  }
}

// The wide form, for launches that leave the GPU idle: there the time is the latency of one
// event's walk, some 5000 instructions in a row, so a block of five warps takes the 32 events of
// a tile.  What does not depend on the frames is computed for all visits at once, a visit per
// warp (mappings and angles; then, with every msq known, masses, momenta and energies); the
// frames follow with a warp per row (a frame step works row by row, and component r of a
// momentum reads row r alone), while the fifth warp multiplies the factor.  Every value comes
// from the same operations in the same order as in phs_event_f64: the same bits.  No friend
// visits (their axis mixes rows).  Slots of a visit (one column per event):
enum {
  kWMsq, kWM,                  // the visited branch
  kWSp, kWCp, kWCt, kWSt,      // its decay angles
  kWFct, kWF, kWA2,            // factors: cos(theta) map; the branch's msq map and (per-event
                               // beams) its constant
  kWPc, kWE0, kWE1, kWRm, kWFk,  // p_decay, daughters' energies, 1/m, sqrt(lambda) / (2 m^2)
  PHS_WIDE_SLOTS
};
#define PHS_WIDE_WARPS 5

template <bool PER_EVENT>
__global__ void __launch_bounds__(PHS_WIDE_WARPS * 32)
    phs_forward_f64_wide_kernel(const __grid_constant__ PhsLaunch a) {
  extern __shared__ double smem[];
  __shared__ unsigned ok_mask;
  const FxRegs k = fx_regs();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const PhsSegment *segs = a.n_segments <= PHS_INLINE_SEGS ? a.seg_inline : a.segments;
  const auto at = [&](int v, int i) -> double & { return smem[(v * PHS_WIDE_SLOTS + i) * 32 + lane]; };
  for (int64_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
    int lo = 0, hi = a.n_segments - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (segs[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    const PhsSegment &seg = segs[lo];
    const int64_t first = (tile - seg.tile_begin) * 32;
    const bool valid = first + lane < seg.ev_count;
    const int64_t local = valid ? first + lane : first;   // (a copy of the tile's first event)
    // checked build: the channel, its slots and the event's rows (block-uniform on the first
    // event; an event out of range writes nothing)
    if (!phs_in(seg.channel, a.n_programs, PHS_CHK_CHANNEL)) continue;
    const PhsChannel &ch = a.channels[seg.channel];
    if (!phs_in(ch.n_visits - 1, a.max_visits, PHS_CHK_VISITS)) continue;
    const bool inside = event_in_bounds(a, seg, local, ch.n_out, ch.n_visits);
    const int64_t ev = seg.ev_begin + local;
    const double *xe = a.x + seg.x_base + local * seg.x_stride;
    double *out = a.p + seg.p_base + local * 4 * (int64_t)ch.n_out;
    const bool lab = PER_EVENT || ch.lab != 0;
    double sqrts = ch.sqrts, lab_bg = ch.lab_bg, lab_ga = ch.lab_gamma;
    if (PER_EVENT) {
      const double E1 = inside ? a.E1[ev] : 1.0, E2 = inside ? a.E2[ev] : 1.0;
      const double r = fx_sqrt(fx_mul(k, E1, E2), k);
      sqrts = fx_add(k, r, r);
      lab_bg = fx_div(fx_sub(k, E1, E2), sqrts, k);
      lab_ga = fx_sqrt(fma(lab_bg, lab_bg, k.one), k);
    }
    const double s = fx_mul(k, sqrts, sqrts);
    const double inv_s = PER_EVENT ? fx_rcp(s, k) : 0.0;
    const int n_visits = ch.n_visits;
    bool ok = true;
    if (threadIdx.x == 0) ok_mask = 0xffffffffu;

    // 1. mappings of each visit's internal daughters, and its angles
    for (int v = wid; v < n_visits; v += PHS_WIDE_WARPS) {
      const PhsVisit &V = ch.visit[v];
      if (v == 0) {
        at(0, kWMsq) = s;
        at(0, kWM) = sqrts;
      }
#pragma unroll 1
      for (int j = 0; j < 2; j++) {
        const PhsChild &C = V.child[j];
        if (!C.internal || !phs_in(V.child_visit[j], n_visits, PHS_CHK_VISITS)) continue;
        double a0 = C.a0, a1 = C.a1, a2 = C.a2, mn = C.msq_min, mx = C.msq_max, mmax = C.m_max;
        if (PER_EVENT) child_constants(k, C, sqrts, ch.m_tot, inv_s, a0, a1, a2, mn, mx, mmax);
        double mq, f, aux;
        map_msq(k, C.map_id, inside ? xrow_at(xe, C.x_msq, seg.x_stride) : 0.5, s, C.m, C.w, mn, mx, a0, a1,
                a2, mq, f, aux);
        const double mj = fx_sqrt(mq, k);
        ok = ok && !fx_gt(mj, mmax);
        const int cv = V.child_visit[j];
        at(cv, kWMsq) = mq;
        at(cv, kWM) = mj;
        at(cv, kWF) = f;
        if (PER_EVENT) at(cv, kWA2) = a2;
      }
      double sp, cp, ct, st, fct, b0 = V.b0, b1 = V.b1;
      sincos2pi(inside ? xrow_at(xe, V.x_phi, seg.x_stride) : 0.5, sp, cp);
      if (PER_EVENT && V.ct_class == PHS_CT_COLLINEAR) {
        b0 = dmul(V.m, V.m) / s;
        b1 = log(dadd(b0, 1.0) / b0);
      }
      map_ct(k, V.ct_class, inside ? xrow_at(xe, V.x_ct, seg.x_stride) : 0.5, b0, b1, ct, st, fct);
      at(v, kWSp) = sp;
      at(v, kWCp) = cp;
      at(v, kWCt) = ct;
      at(v, kWSt) = st;
      at(v, kWFct) = fct;
    }
    __syncthreads();

    // 2. kinematics of each visit
    for (int v = wid; v < n_visits; v += PHS_WIDE_WARPS) {
      const PhsVisit &V = ch.visit[v];
      double cmsq[2], cm[2];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const bool in = V.child[j].internal && phs_in(V.child_visit[j], n_visits, PHS_CHK_VISITS);
        cmsq[j] = in ? at(V.child_visit[j], kWMsq) : V.child[j].msq_leaf;
        cm[j] = in ? at(V.child_visit[j], kWM) : V.child[j].m_leaf;
      }
      const double msq_b = at(v, kWMsq), m_b = at(v, kWM);
      const int massless = V.massless;
      double sl;
      ok = kallen_ok(k, massless, msq_b, m_b, cmsq, cm, sl) && ok;
      double rm = 0.0, pc, ce0, ce1;
      if (massless == 3) {
        pc = ce0 = ce1 = fx_scale(m_b, -1);
        if (V.kind == PHS_KIND_ROOT) rm = fx_hi(m_b) - 1u < 0x7fefffffu ? fx_rcp(m_b, k) : 0.0;   // n_out = 2
      } else {
        double hm;
        if (!PER_EVENT && V.self_root) {
          rm = ch.inv_sqrts;
          hm = fx_scale(rm, -1);
        } else {
          mass_reciprocals(k, m_b, rm, hm);
        }
        pc = fx_mul(k, sl, hm);
        at(v, kWFk) = fx_mul(k, pc, rm);
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
      at(v, kWPc) = pc;
      at(v, kWE0) = ce0;
      at(v, kWE1) = ce1;
      at(v, kWRm) = rm;
    }
    const unsigned mine = __ballot_sync(0xffffffffu, ok && valid);
    if (lane == 0) atomicAnd(&ok_mask, mine);
    __syncthreads();
    const unsigned passed = ok_mask;
    ok = passed >> lane & 1;

    // 3. the factor (warp 4), and the frames and momenta, row `wid` (warps 0 .. 3)
    if (wid == 4) {
      double factor = PER_EVENT ? 1.0 : ch.f0;
      int halved = 0;
      for (int v = 0; v < n_visits && passed; v++) {
        const PhsVisit &V = ch.visit[v];
        for (int j = 0; j < 2; j++) {
          const PhsChild &C = V.child[j];
          if (!C.internal || !phs_in(V.child_visit[j], n_visits, PHS_CHK_VISITS)) continue;
          if (PER_EVENT && C.map_id != PHS_MAP_STEP_E && C.map_id != PHS_MAP_STEP_H)
            factor = fx_mul(k, factor, at(V.child_visit[j], kWA2));
          if (C.map_id != PHS_MAP_NO) factor = fx_mul(k, factor, at(V.child_visit[j], kWF));
        }
        if (V.massless != 3) {
          factor = fx_mul(k, factor, at(v, kWFk));
          halved++;
        }
        if (V.ct_class == PHS_CT_COLLINEAR) factor = fx_mul(k, factor, at(v, kWFct));
      }
      if (valid && inside) {
        a.volume[ev] = PER_EVENT ? channel_volume(ch, sqrts) : ch.volume;
        a.factor[ev * a.factor_stride + seg.factor_col] =
            ok ? fx_mul(k, factor, fx_double((1023u + halved) << 20, 0u)) : 0.0;
        a.ok[ev] = ok ? 1 : 0;
      }
    } else if (passed == 0) {
      if (valid && inside)
        for (int i = 0; i < ch.n_out; i++) out[4 * i + wid] = 0.0;
    } else {
      const bool first_row = wid == 0, edge = wid == 0 || wid == 3;
      double l[4] = {0.0, 0.0, 0.0, 0.0}, s0[4] = {}, s1[4] = {};   // the row, and saved ones
      int sp = 0;
      const auto put = [&](int index, double q) {
        if (valid && inside && phs_in(index, ch.n_out, PHS_CHK_P)) out[4 * index + wid] = ok ? q : 0.0;
      };
      for (int v = 0; v < n_visits; v++) {
        const PhsVisit &V = ch.visit[v];
        int kind = V.kind;
        if (lab)
          kind = kind == PHS_KIND_ROOT ? PHS_KIND_ROOT_LAB
                 : kind == PHS_KIND_FIRST ? PHS_KIND_FIRST_LAB
                 : kind == PHS_KIND_LEAVES_FIRST ? PHS_KIND_LEAVES : kind;
        const bool pair = kind == PHS_KIND_LEAVES || kind == PHS_KIND_LEAVES_FIRST;
        // the branch's momentum and energy in its parent's frame
        double p_b = 0.0, E_b = 0.0;
        if (phs_in(V.parent_visit + 1, n_visits + 1, PHS_CHK_VISITS) && V.parent_visit >= 0) {
          const double pp = at(V.parent_visit, kWPc);
          p_b = V.parent_child == 0 ? pp : fx_neg(pp);
          E_b = at(V.parent_visit, V.parent_child == 0 ? kWE0 : kWE1);
        }
        const double pc = at(v, kWPc), ce0 = at(v, kWE0), ce1 = at(v, kWE1), rm = at(v, kWRm);
        Step t;
        t.sp = at(v, kWSp);
        t.cp = at(v, kWCp);
        t.ct = at(v, kWCt);
        t.st = at(v, kWSt);
        if (pair) {
          const double pst = fx_mul(k, pc, t.st), qx = fx_mul(k, pst, t.cp), qy = fx_mul(k, pst, t.sp);
          double qa0, qa3, qb0, qb3;
          if (V.massless == 3) {
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
          double qa, qb;
          if (kind == PHS_KIND_LEAVES_FIRST) {
            const double w = wid == 3 ? fx_mul(k, l[1], qx) : fma(l[2], qy, fx_mul(k, l[1], qx));
            qa = first_row ? qa0 : fma(l[3], qa3, w);
            qb = first_row ? qb0 : fma(l[3], qb3, -w);
          } else {
            const double w = fma(l[2], qy, fx_mul(k, l[1], qx));
            qa = fma(l[0], qa0, fma(l[3], qa3, w));
            qb = fma(l[0], qb0, fma(l[3], qb3, -w));
          }
          put(V.child[0].out_index, qa);
          put(V.child[1].out_index, qb);
        } else {
          if (!V.self_root) {
            t.bg = fx_mul(k, p_b, rm);
            t.ga = fx_mul(k, E_b, rm);
          }
          if (kind == PHS_KIND_ROOT || kind == PHS_KIND_ROOT_LAB) {
            if (edge) {
              const double g = kind == PHS_KIND_ROOT ? (first_row ? 1.0 : 0.0) : (first_row ? lab_ga : lab_bg);
              const double h = kind == PHS_KIND_ROOT ? (first_row ? 0.0 : 1.0) : (first_row ? lab_bg : lab_ga);
              l[0] = g;
              l[1] = fx_mul(k, -h, t.st);
              l[2] = 0.0;
              l[3] = fx_mul(k, h, t.ct);
            } else {
              const double c = wid == 1 ? t.cp : t.sp;
              l[0] = 0.0;
              l[1] = fx_mul(k, t.ct, c);
              l[2] = wid == 1 ? fx_neg(t.sp) : t.cp;
              l[3] = fx_mul(k, t.st, c);
            }
          } else if (kind == PHS_KIND_FIRST) {
            if (first_row) {
              l[0] = t.ga;
              l[1] = fx_mul(k, -t.st, t.bg);
              l[2] = 0.0;
              l[3] = fx_mul(k, t.ct, t.bg);
            } else if (wid == 3) {
              frame_row<true, true>(k, t, l);
            } else {
              frame_row<true, false>(k, t, l);
            }
          } else if (kind == PHS_KIND_FIRST_LAB) {
            if (edge) frame_row<false, true>(k, t, l); else frame_row<true, false>(k, t, l);
          } else {
            frame_row<false, false>(k, t, l);
          }
          for (int j = 0; j < 2; j++)
            if (!V.child[j].internal)
              put(V.child[j].out_index, fma(l[0], j == 0 ? ce0 : ce1, fx_mul(k, l[3], j == 0 ? pc : fx_neg(pc))));
        }
        if (V.push >= 0) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            if (sp == 0) s0[i] = l[i]; else s1[i] = l[i];
          }
          sp++;
        }
        if (V.carry < 0 && sp > 0) {
          sp--;
#pragma unroll
          for (int i = 0; i < 4; i++) l[i] = sp == 0 ? s0[i] : s1[i];
        }
      }
    }
    __syncthreads();   // the slots are read
  }
}

// Whizard's sparse momentum buffer from the dense one (layout in phs_device.h): one thread
// per 32-byte slot, consecutive threads on consecutive slots.
__global__ void phs_whizard_sparse_kernel(const __grid_constant__ PhsSparseLaunch a) {
  const int64_t total = a.n_events * a.n_prt;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ev = i / a.n_prt;
    const int code = (int)(i - ev * a.n_prt) + 1;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const double *pe = a.p + ev * 4 * a.n_out;
    if (code < (1 << a.n_out)) {
      if ((code & (code - 1)) == 0) {
        const int k = __ffs(code) - 1;
#pragma unroll
        for (int mu = 0; mu < 4; mu++) v[mu] = pe[4 * k + mu];
      } else if (a.internal[code >> 5] >> (code & 31) & 1u) {
        // back to the centre-of-mass frame: the inverse of the lab boost
        // p0 = gamma p0* + bg p3*, p3 = bg p0* + gamma p3* (phs.cu:1286-1301)
        const double e1 = a.E1 ? a.E1[ev] : a.e1, e2 = a.E2 ? a.E2[ev] : a.e2;
        const double bg = (e1 - e2) / (2.0 * sqrt(e1 * e2)), ga = sqrt(1.0 + bg * bg);
        for (int k = 0; k < a.n_out; k++) {
          if (!(code >> k & 1)) continue;
          const double *q = pe + 4 * k;
          v[0] += ga * q[0] - bg * q[3];
          v[1] += q[1];
          v[2] += q[2];
          v[3] += ga * q[3] - bg * q[0];
        }
      }
    }
    double2 *o = reinterpret_cast<double2 *>(a.out + 4 * i);
    o[0] = make_double2(v[0], v[1]);
    o[1] = make_double2(v[2], v[3]);
  }
}

// Philox4x32-10 (Salmon et al., SC'11); layout documented in gpu_phs_gb300/philox.py.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

__global__ void phs_philox_kernel(double *x, int64_t e0, int64_t n, uint64_t seed) {
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const int64_t b_first = e0 >> 1, b_last = (e0 + n - 1) >> 1;
  for (int64_t b = b_first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= b_last;
       b += (int64_t)gridDim.x * blockDim.x) {
    uint4 r = philox4x32_10(make_uint4((uint32_t)b, (uint32_t)((uint64_t)b >> 32), 0u, 0u), key);
    const double u0 = (double)((((uint64_t)r.x << 32) | r.y) >> 11) * 0x1.0p-53;
    const double u1 = (double)((((uint64_t)r.z << 32) | r.w) >> 11) * 0x1.0p-53;
    const int64_t e = 2 * b;
    if (e >= e0 && e < e0 + n) x[e - e0] = u0;
    if (e + 1 >= e0 && e + 1 < e0 + n) x[e + 1 - e0] = u1;
  }
}

// Arithmetic-throughput probe: each thread runs `iters` rounds of 8 independent FMA
// chains (FP64 or FP32), enough independent work to keep the pipe busy; the result is
// stored so the chains are live.
template <typename T>
__global__ void phs_fma_rate_kernel(T *out, int iters, T a, T b) {
  T v[8];
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = (T)(threadIdx.x + i);
  for (int k = 0; k < iters; k++) {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = fma(v[i], a, b);
  }
  T s = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) s += v[i];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace

cudaError_t phs_launch_fma_rate(void *out, int fp64, int blocks, int threads, int iters,
                                cudaStream_t stream) {
  if (fp64)
    phs_fma_rate_kernel<double><<<blocks, threads, 0, stream>>>((double *)out, iters, 0.999999, 1e-7);
  else
    phs_fma_rate_kernel<float><<<blocks, threads, 0, stream>>>((float *)out, iters, 0.999999f, 1e-7f);
  return cudaGetLastError();
}

size_t phs_forward_smem_bytes(int stack_depth, int block) {
  // frame stack, the compacting variant's per-warp queues (64 events per warp)
  return (size_t)stack_depth * PHS_STATE * block * sizeof(double) +
         (size_t)(block / 32) * 64 * sizeof(int64_t);
}

// Variants (each at one block shape, BLOCK threads, and a register budget): 0: one pass,
// 128 threads x 4 blocks per SM; 1, 2: compacting, 128 x 4 and 128 x 3 (no spills);
// 3, 4: one pass, 256 x 2 and 64 x 8; 5-8: split (the FP32 pre-test, then the walk over its
// survivors; uniform beams only), 128 x 4, 128 x 3, 256 x 2, 64 x 8.  The 128-register
// budget is the same for 64 x 8, 128 x 4 and 256 x 2.
static int f64_block(int variant) {
  switch (variant) {
    case 3: case 7: return 256;
    case 4: case 8: return 64;
    default: return PHS_FWD_BLOCK;
  }
}

template <bool PER_EVENT>
static const void *f64_kernel(int variant) {
  switch (variant) {
    case 1: return (const void *)phs_forward_f64_kernel<PER_EVENT, true, 4>;
    case 2: return (const void *)phs_forward_f64_kernel<PER_EVENT, true, 3>;
    case 3: return (const void *)phs_forward_f64_kernel<PER_EVENT, false, 2, 256>;
    case 4: return (const void *)phs_forward_f64_kernel<PER_EVENT, false, 8, 64>;
    case 5: return (const void *)phs_f64_walk_kernel<4>;
    case 6: return (const void *)phs_f64_walk_kernel<3>;
    case 7: return (const void *)phs_f64_walk_kernel<2, 256>;
    case 8: return (const void *)phs_f64_walk_kernel<8, 64>;
    default: return (const void *)phs_forward_f64_kernel<PER_EVENT, false, 4>;
  }
}

int phs_forward_block_size(int variant) { return f64_block(variant); }

// Shared memory above the 48 KB default (256-thread blocks with two saved frames) needs
// the kernel's opt-in.
static cudaError_t allow_smem(const void *kernel, size_t smem) {
  if (smem <= 48 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

int phs_forward_blocks_per_sm(int stack_depth, bool per_event, int variant) {
  int n = 0;
  const int block = f64_block(variant);
  const size_t smem = phs_forward_smem_bytes(stack_depth, block);
  const void *k = per_event ? f64_kernel<true>(variant) : f64_kernel<false>(variant);
  if (allow_smem(k, smem) != cudaSuccess) return 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, block, smem);
  return n > 0 ? n : 1;
}

template <bool PER_EVENT>
static cudaError_t launch_wide(const PhsLaunch &a, cudaStream_t stream) {
  const size_t smem = (size_t)a.max_visits * PHS_WIDE_SLOTS * 32 * sizeof(double);
  const cudaError_t e = allow_smem((const void *)phs_forward_f64_wide_kernel<PER_EVENT>, smem);
  if (e != cudaSuccess) return e;
  const int64_t cap = 1 << 20;
  phs_forward_f64_wide_kernel<PER_EVENT>
      <<<(int)(a.n_tiles < cap ? a.n_tiles : cap), PHS_WIDE_WARPS * 32, smem, stream>>>(a);
  return cudaGetLastError();
}

template <bool PER_EVENT>
static cudaError_t launch_f64(const PhsLaunch &a, int n_blocks, int variant, cudaStream_t stream) {
  const int block = f64_block(variant);
  const size_t smem = phs_forward_smem_bytes(a.stack_depth, block);
  const cudaError_t e = allow_smem(f64_kernel<PER_EVENT>(variant), smem);
  if (e != cudaSuccess) return e;
  switch (variant) {
    case 1:
      phs_forward_f64_kernel<PER_EVENT, true, 4><<<n_blocks, block, smem, stream>>>(a);
      break;
    case 2:
      phs_forward_f64_kernel<PER_EVENT, true, 3><<<n_blocks, block, smem, stream>>>(a);
      break;
    case 3:
      phs_forward_f64_kernel<PER_EVENT, false, 2, 256><<<n_blocks, block, smem, stream>>>(a);
      break;
    case 4:
      phs_forward_f64_kernel<PER_EVENT, false, 8, 64><<<n_blocks, block, smem, stream>>>(a);
      break;
    default:
      phs_forward_f64_kernel<PER_EVENT, false, 4><<<n_blocks, block, smem, stream>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t phs_launch_forward_f64(const PhsLaunch &a, int n_blocks, int variant,
                                   cudaStream_t stream) {
  if (a.n_tiles <= 0) return cudaSuccess;
  if (variant == PHS_F64_WIDE) {
    if (a.friends) return cudaErrorInvalidValue;
    return a.E1 && a.E2 ? launch_wide<true>(a, stream) : launch_wide<false>(a, stream);
  }
  if (variant >= 5) {
    if (a.E1 || a.E2) return cudaErrorInvalidValue;  // the pre-test needs uniform beams
    cudaError_t e = phs_launch_pretest(a, stream);
    if (e != cudaSuccess) return e;
    const int block = f64_block(variant);
    const size_t smem = phs_forward_smem_bytes(a.stack_depth, block);
    e = allow_smem(f64_kernel<false>(variant), smem);
    if (e != cudaSuccess) return e;
    switch (variant) {
      case 5: phs_f64_walk_kernel<4><<<n_blocks, block, smem, stream>>>(a); break;
      case 6: phs_f64_walk_kernel<3><<<n_blocks, block, smem, stream>>>(a); break;
      case 7: phs_f64_walk_kernel<2, 256><<<n_blocks, block, smem, stream>>>(a); break;
      default: phs_f64_walk_kernel<8, 64><<<n_blocks, block, smem, stream>>>(a);
    }
    return cudaGetLastError();
  }
  return a.E1 && a.E2 ? launch_f64<true>(a, n_blocks, variant, stream)
                      : launch_f64<false>(a, n_blocks, variant, stream);
}

// SMs of the current device (grid caps of the grid-stride kernels below).
static int current_sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

cudaError_t phs_launch_whizard_sparse(const PhsSparseLaunch &a, cudaStream_t stream) {
  const int64_t total = a.n_events * a.n_prt;
  if (total <= 0) return cudaSuccess;
  const int64_t blocks = (total + 255) / 256, cap = (int64_t)current_sm_count() * 32;
  phs_whizard_sparse_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, stream>>>(a);
  return cudaGetLastError();
}

cudaError_t phs_launch_philox(double *x, int64_t n_events, int32_t n_x, uint64_t seed,
                              int64_t first_event, cudaStream_t stream) {
  const int64_t n = n_events * n_x;
  if (n <= 0) return cudaSuccess;
  const int64_t blocks_needed = ((n >> 1) + 2 + 255) / 256, cap = (int64_t)current_sm_count() * 16;
  const int grid = (int)(blocks_needed < cap ? blocks_needed : cap);
  phs_philox_kernel<<<grid, 256, 0, stream>>>(x, first_event * n_x, n, seed);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Forward generation without device allocation.
//
// For callers that must not allocate device memory: code running inside a host that
// owns the device heap through its own allocator, sandboxes or plugins denied cudaMalloc,
// and drivers that would otherwise synchronise the device inside their hot loop.  The
// channel programs and the segment table, which the regular entry points keep in buffers
// the library allocates, live here in one file-scope device array instead.  Every GPU
// that loads the library holds this array (sizeof(PhsNoAllocScratch), about 1 MB) until
// the process exits.  All calls share it and it keeps the last call's contents; each call
// overwrites everything it reads, so nothing needs clearing, but calls that overlap on
// the GPU (different streams or host threads) race on it.
struct PhsNoAllocScratch {
  PhsChannel channels[PHS_NOALLOC_MAX_CHANNELS];
  PhsSegment segments[PHS_NOALLOC_MAX_CHANNELS];
};

static __device__ __align__(256) unsigned char phs_noalloc_scratch[sizeof(PhsNoAllocScratch)];

// Device address of the scratch array per device (filled at set-up; in host code the
// array's name only stands in for the symbol and is never a device address).  The mutex
// orders first calls from several host threads.
static void *g_noalloc_addr[256];
static std::mutex g_noalloc_mu;

size_t phs_noalloc_scratch_bytes() { return sizeof(PhsNoAllocScratch); }

cudaError_t phs_launch_forward_f64_noalloc(PhsLaunch a, const PhsChannel *channels,
                                           int n_channels, const PhsSegment *segments,
                                           int n_segments, int n_blocks, cudaStream_t stream) {
  if (n_channels > PHS_NOALLOC_MAX_CHANNELS || n_segments > PHS_NOALLOC_MAX_CHANNELS)
    return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
  void *addr = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      // set-up, once per device, with that device current
      void *ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, phs_noalloc_scratch);
      if (e != cudaSuccess) return e;
      g_noalloc_addr[dev] = ptr;
    }
    addr = g_noalloc_addr[dev];
  }
  PhsNoAllocScratch *s = static_cast<PhsNoAllocScratch *>(addr);
  // pageable host sources: each copy has read its source when the call returns
  e = cudaMemcpyAsync(s->channels, channels, (size_t)n_channels * sizeof(PhsChannel),
                      cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return e;
  if (n_segments > 0) {
    e = cudaMemcpyAsync(s->segments, segments, (size_t)n_segments * sizeof(PhsSegment),
                        cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
  }
  a.channels = s->channels;
  a.segments = s->segments;
  a.n_segments = n_segments;
  if (a.n_tiles <= 0) return cudaSuccess;
  const size_t smem = phs_forward_smem_bytes(a.stack_depth, PHS_FWD_BLOCK);
  e = allow_smem(f64_kernel<false>(0), smem);
  if (e != cudaSuccess) return e;
  phs_forward_f64_kernel<false, false, 4><<<n_blocks, PHS_FWD_BLOCK, smem, stream>>>(a);
  return cudaGetLastError();
}

PHS_CHECK_COLLECTOR(phs_check_collect_kernels)
