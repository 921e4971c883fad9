// phs_pretest.h -- msq of one branch in plain FP32 with an error bound, for the FP32 pre-test
// (host and device; tests/test_pretest_host.py checks the bound with the hardware functions' errors
// at their limits).
#pragma once
#include <math.h>
#include <stdint.h>

#include "phs_fix.h"
#include "phs_program.h"

#if defined(__CUDA_ARCH__)
FX_FN float pt_sin(float a) { return __sinf(a); }
FX_FN float pt_cos(float a) { return __cosf(a); }
FX_FN float pt_exp(float a) { return __expf(a); }
FX_FN float pt_div(float a, float b) { return __fdividef(a, b); }
#else
FX_FN float pt_sin(float a) { return sinf(a); }
FX_FN float pt_cos(float a) { return cosf(a); }
FX_FN float pt_exp(float a) { return expf(a); }
FX_FN float pt_div(float a, float b) { return a / b; }
#endif

// The bound: 64 epsilons (3.8e-6 = k) times the magnitudes of the terms that msq is made of.  Per
// unit of the magnitudes: the angle w of the tangent is within 5e-7 (x, the constants, product and
// sum, rounded to nearest, of magnitudes up to pi), the hardware sine and cosine within 2^-21.4 and
// 2^-21.2 (|w| <= pi/4), so tan or cot within 1.3e-6 (1 + tan^2); the hardware exponential within 2 +
// 1.2 |y| epsilons, its argument within 3 epsilons of |y|.
// These are first order: a cotangent 1/w' - 1/w = (w - w') / (w w') is within k (1 + 1/w'^2) only
// while w - w' <= k w / w', that is while w' is not many times w.  Next to pi/2 (a resonance of width
// m Gamma << s, x at its end) w itself is down to m Gamma / s, so w has to be right to a few per cent
// of itself: 1 - x is formed from all of x's bits (within 2^-49), and a sine below 2^-8 is its
// argument (within 3e-6 of itself, which 1/w >= 256 makes 1e-3 of the bound).
#define PHS_F32_EPS_BOUND (64.0f * 5.9604645e-8f)

// A double to the nearest float (ties away) with integer operations: the conversion unit for
// doubles takes 16 cycles of an SM a warp.  Below 2^-126: 0; for |d| < 2^128.
FX_FN float f32_of(double d) {
  const uint64_t b = fx_bits(d) + 0x10000000ull;
  const uint32_t hw = (uint32_t)(b >> 32), mag = hw & 0x7fffffffu;
  return mag < (897u << 20) ? 0.0f
                            : fx_float((hw & 0x80000000u) | ((mag - (896u << 20)) << 3) | ((uint32_t)b >> 29));
}
// 1 - d for 0 <= d <= 1, x = f32_of(d): within 2^-49 for d >= 0.5 (1 - x is exact, and what x left of
// d, 29 bits with their sign, is in units of 2^-53), 2^-23 of itself below.
FX_FN float f32_one_minus(double d, float x) {
  const int32_t rest = (int32_t)(fx_lo(d) << 3) >> 3;
  return fx_fmaf((float)rest, -0x1p-53f, 1.0f - x);
}

// msq at x = xd and the bound e on its error; c0..c5: the packed constants of PhsTestChild.
FX_FN float msq_f32(int map_id, float c0, float c1, float c2, float c3, float c4, float c5, double xd, float &e) {
  const float x = f32_of(xd), k = PHS_F32_EPS_BOUND;
  switch (map_id) {
    case PHS_MAP_NO:
      e = k * (fabsf(c0) + fabsf(c1));
      return c0 + x * (c1 - c0);
    case PHS_MAP_SCHANNEL: {
      // one tangent per lane, of z or of pi/2 -+ z (selected, not branched: lanes of a warp
      // take different sides)
      const float z = c0 + x * c1;  // c1 holds a1 - a0
      const bool hi_side = z > 0.78539816f, lo_side = z < -0.78539816f, cot = hi_side || lo_side;
      const float w = hi_side ? c3 + f32_one_minus(xd, x) * c1 : (lo_side ? c2 + x * c1 : z);
      const float sw = fabsf(w) < 0x1p-8f ? w : pt_sin(w), cw = pt_cos(w);
      const float q = pt_div(cot ? cw : sw, cot ? sw : cw), t = lo_side ? -q : q;
      e = k * (fabsf(c4) + fabsf(c5) * (1.0f + t * t));
      return c4 + c5 * t;
    }
    case PHS_MAP_COLLINEAR:
    case PHS_MAP_INFRARED:
    case PHS_MAP_RADIATION:
    case PHS_MAP_TCHANNEL:
    case PHS_MAP_UCHANNEL: {
      const bool upper = (map_id == PHS_MAP_TCHANNEL || map_id == PHS_MAP_UCHANNEL) && !(xd < 0.5);
      const float y = (upper ? f32_one_minus(xd, x) : x) * c1, em = pt_exp(y) - 1.0f;
      e = k * (fabsf(upper ? c3 : c2) + fabsf(c0) * (em + 1.0f) * (1.0f + fabsf(y)));
      return upper ? c3 - c0 * em : c0 * em + c2;
    }
  }
  e = INFINITY;
  return 0.0f;
}
