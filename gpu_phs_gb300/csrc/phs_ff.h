// phs_ff.h -- float-float ("FP32 pair") arithmetic for the FP32-pipe forward kernel.
//
// A value is hi + lo with two floats, |lo| <= ulp(hi)/2, about 48 significant bits.  The
// primitives are the error-free transformations of Knuth (TwoSum) and Dekker (Fast2Sum,
// and the product via FMA), composed as in Dekker, "A floating-point technique for
// extending the available precision", Numer. Math. 18 (1971).  Arithmetic goes through
// explicit round-to-nearest intrinsics so no compiler contraction or reassociation can
// break an error-free step.  The elementary functions reduce their argument with a table
// of exact multiples (kept in shared memory by the kernel) and evaluate short Taylor
// series; leading terms in float-float, the small tail in plain float.  Accuracy against
// long double on the host: 3e-14 relative for the arithmetic, 6e-15 absolute for sin and
// cos, 1.5e-13 relative for exp, 3e-14 relative for tan up to pi/4 (3.7e-13 within 0.04 of
// pi/2, where the callers take the cotangent of the complement), far inside what the forward
// map needs for momenta within 1e-6.
//
// The header also compiles as host C++ (for CPU validation of the functions).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FF_FN __host__ __device__ __forceinline__
#else
#define FF_FN inline
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
#endif

struct ff {
  float hi, lo;
};

#if defined(__CUDA_ARCH__)
FF_FN float f_add(float a, float b) { return __fadd_rn(a, b); }
FF_FN float f_sub(float a, float b) { return __fsub_rn(a, b); }
FF_FN float f_mul(float a, float b) { return __fmul_rn(a, b); }
FF_FN float f_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
#else
FF_FN float f_add(float a, float b) { volatile float r = a + b; return r; }
FF_FN float f_sub(float a, float b) { volatile float r = a - b; return r; }
FF_FN float f_mul(float a, float b) { volatile float r = a * b; return r; }
FF_FN float f_fma(float a, float b, float c) { return fmaf(a, b, c); }
#endif

FF_FN ff ff_make(float hi, float lo) { ff r; r.hi = hi; r.lo = lo; return r; }
FF_FN ff ff_from_float(float a) { return ff_make(a, 0.0f); }

// Fast2Sum: |a| >= |b| (or a == 0).
FF_FN ff fast_two_sum(float a, float b) {
  float s = f_add(a, b);
  float e = f_sub(b, f_sub(s, a));
  return ff_make(s, e);
}

// TwoSum: any a, b.
FF_FN ff two_sum(float a, float b) {
  float s = f_add(a, b);
  float bb = f_sub(s, a);
  float e = f_add(f_sub(a, f_sub(s, bb)), f_sub(b, bb));
  return ff_make(s, e);
}

FF_FN ff two_prod(float a, float b) {
  float p = f_mul(a, b);
  float e = f_fma(a, b, -p);
  return ff_make(p, e);
}

FF_FN ff ff_neg(ff a) { return ff_make(-a.hi, -a.lo); }

FF_FN ff ff_add(ff a, ff b) {
  ff s = two_sum(a.hi, b.hi);
  float e = f_add(s.lo, f_add(a.lo, b.lo));
  return fast_two_sum(s.hi, e);
}

FF_FN ff ff_sub(ff a, ff b) { return ff_add(a, ff_neg(b)); }

FF_FN ff ff_add_f(ff a, float b) {
  ff s = two_sum(a.hi, b);
  float e = f_add(s.lo, a.lo);
  return fast_two_sum(s.hi, e);
}

FF_FN ff ff_mul(ff a, ff b) {
  ff p = two_prod(a.hi, b.hi);
  float e = f_fma(a.hi, b.lo, p.lo);
  e = f_fma(a.lo, b.hi, e);
  return fast_two_sum(p.hi, e);
}

FF_FN ff ff_mul_f(ff a, float b) {
  ff p = two_prod(a.hi, b);
  float e = f_fma(a.lo, b, p.lo);
  return fast_two_sum(p.hi, e);
}

FF_FN ff ff_sqr(ff a) {
  ff p = two_prod(a.hi, a.hi);
  float e = f_fma(f_add(a.hi, a.hi), a.lo, p.lo);
  return fast_two_sum(p.hi, e);
}

#if defined(__CUDA_ARCH__)
FF_FN float f_rcp_approx(float a) { return __fdividef(1.0f, a); }   // hardware approximation
FF_FN float f_rsqrt_approx(float a) { return rsqrtf(a); }
#else
FF_FN float f_rcp_approx(float a) { return 1.0f / a; }
FF_FN float f_rsqrt_approx(float a) { return 1.0f / sqrtf(a); }
#endif

// 1/b: the hardware reciprocal estimate refined by one Newton step with the residual
// 1 - b y in float-float (~2^-44 relative).
FF_FN ff ff_recip_fast(ff b) {
  const float y = f_rcp_approx(b.hi);
  const ff p = two_prod(b.hi, y);
  const float e = f_sub(f_sub(f_sub(1.0f, p.hi), p.lo), f_mul(b.lo, y));
  return fast_two_sum(y, f_mul(y, e));
}

// a/b with the reciprocal estimate: q1 = a.hi y, then one correction from a - b q1 (its leading
// difference is exact: b q1 lies within a few ulps of a).
FF_FN ff ff_div_fast(ff a, ff b) {
  const float y = f_rcp_approx(b.hi);
  const float q1 = f_mul(a.hi, y);
  const ff p = two_prod(b.hi, q1);
  const float r = f_add(f_sub(a.hi, p.hi), f_sub(a.lo, f_fma(b.lo, q1, p.lo)));
  return fast_two_sum(q1, f_mul(r, y));
}

// sqrt(a), a >= 0, from the hardware rsqrt estimate and one Newton step in float-float (the
// residual as in ff_div_fast).
FF_FN ff ff_sqrt_fast(ff a) {
  if (!(a.hi > 0.0f)) return ff_make(0.0f, 0.0f);
  const float y = f_rsqrt_approx(a.hi);
  const float s = f_mul(a.hi, y);
  const ff p = two_prod(s, s);
  const float r = f_add(f_sub(a.hi, p.hi), f_sub(a.lo, p.lo));
  return fast_two_sum(s, f_mul(f_mul(r, y), 0.5f));
}

// a0 b0 + a1 b1 (+ a2 b2 + a3 b3): exact products of the high parts summed with TwoSum,
// every rounding error and cross term gathered in one float, one normalization at the end.
FF_FN ff ff_dot2(ff a0, ff b0, ff a1, ff b1) {
  const ff p0 = two_prod(a0.hi, b0.hi), p1 = two_prod(a1.hi, b1.hi);
  float e = f_fma(a0.hi, b0.lo, f_fma(a0.lo, b0.hi, p0.lo));
  e = f_add(e, f_fma(a1.hi, b1.lo, f_fma(a1.lo, b1.hi, p1.lo)));
  const ff s = two_sum(p0.hi, p1.hi);
  return fast_two_sum(s.hi, f_add(e, s.lo));
}

// The same without the final normalization (|lo| may reach a few ulps of hi): for a value that
// is widened to a double next.
FF_FN ff ff_dot2_raw(ff a0, ff b0, ff a1, ff b1) {
  const ff p0 = two_prod(a0.hi, b0.hi), p1 = two_prod(a1.hi, b1.hi);
  float e = f_fma(a0.hi, b0.lo, f_fma(a0.lo, b0.hi, p0.lo));
  e = f_add(e, f_fma(a1.hi, b1.lo, f_fma(a1.lo, b1.hi, p1.lo)));
  const ff s = two_sum(p0.hi, p1.hi);
  return ff_make(s.hi, f_add(e, s.lo));
}

// a0 b0 + a1 b1 + c, not normalized.
FF_FN ff ff_dot2_add_raw(ff a0, ff b0, ff a1, ff b1, ff c) {
  const ff p0 = two_prod(a0.hi, b0.hi), p1 = two_prod(a1.hi, b1.hi);
  float e = f_fma(a0.hi, b0.lo, f_fma(a0.lo, b0.hi, p0.lo));
  e = f_add(e, f_fma(a1.hi, b1.lo, f_fma(a1.lo, b1.hi, p1.lo)));
  e = f_add(e, c.lo);
  ff s = two_sum(p0.hi, p1.hi);
  e = f_add(e, s.lo);
  s = two_sum(s.hi, c.hi);
  return ff_make(s.hi, f_add(e, s.lo));
}

FF_FN ff ff_dot3(ff a0, ff b0, ff a1, ff b1, ff a2, ff b2) {
  const ff p0 = two_prod(a0.hi, b0.hi), p1 = two_prod(a1.hi, b1.hi);
  const ff p2 = two_prod(a2.hi, b2.hi);
  float e = f_fma(a0.hi, b0.lo, f_fma(a0.lo, b0.hi, p0.lo));
  e = f_add(e, f_fma(a1.hi, b1.lo, f_fma(a1.lo, b1.hi, p1.lo)));
  e = f_add(e, f_fma(a2.hi, b2.lo, f_fma(a2.lo, b2.hi, p2.lo)));
  ff s = two_sum(p0.hi, p1.hi);
  e = f_add(e, s.lo);
  s = two_sum(s.hi, p2.hi);
  return fast_two_sum(s.hi, f_add(e, s.lo));
}

#if defined(__CUDA_ARCH__)
FF_FN uint64_t ff_dbits(double d) { return (uint64_t)__double_as_longlong(d); }
FF_FN double ff_bitsd(uint64_t b) { return __longlong_as_double((long long)b); }
FF_FN uint32_t ff_fbits(float f) { return __float_as_uint(f); }
FF_FN float ff_bitsf(uint32_t b) { return __uint_as_float(b); }
FF_FN int ff_clz(uint32_t v) { return __clz((int)v); }
#else
FF_FN uint64_t ff_dbits(double d) { uint64_t b; memcpy(&b, &d, 8); return b; }
FF_FN double ff_bitsd(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
FF_FN uint32_t ff_fbits(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
FF_FN float ff_bitsf(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
FF_FN int ff_clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
#endif

// Double -> float-float (48 bits) without FP64 instructions: the significand's upper 24 bits are the high
// part's, the 29 bits below it are converted as an integer and scaled (rounded to 24 bits).  The
// high part is truncated, so for 0 <= d < 1 the order against 0.5 is kept exactly (d < 0.5 iff
// hi < 0.5f).  Values below 2^-103 in magnitude (or non-finite) are not handled: their low part
// reads as 0.
FF_FN ff ff_from_double_int(double d) {
  const uint64_t b = ff_dbits(d);
  const uint32_t hw = (uint32_t)(b >> 32), lw = (uint32_t)b, sign = hw & 0x80000000u;
  const uint32_t mag = hw & 0x7fffffffu;
  if (mag < (897u << 20)) return ff_make(0.0f, 0.0f);           // below 2^-126
  const uint32_t hi = sign | ((mag - (896u << 20)) << 3) | (lw >> 29);
  // the low field has weight 2^(e - 52), e the unbiased exponent: r 2^-29 2^(e - 23)
  const int fe = (int)(mag >> 20) - 919;
  const float scale = ff_bitsf(fe > 0 ? sign | ((uint32_t)fe << 23) : 0u);
  return ff_make(ff_bitsf(hi), f_mul(f_mul((float)(lw & 0x1fffffffu), 0x1p-29f), scale));
}

// D * 2^e2 for an integer 0 < D < 2^63, truncated to 48 bits, with integer operations only.
FF_FN ff ff_from_mantissa(uint64_t D, int e2) {
  const uint32_t dh = (uint32_t)(D >> 32), dl = (uint32_t)D;
  const int p = dh ? 63 - ff_clz(dh) : 31 - ff_clz(dl);   // leading one of D
  const int fe = p + e2 + 127;
  if (fe < 1) return ff_make(0.0f, 0.0f);
  const uint32_t mh = p >= 23 ? (uint32_t)(D >> (p - 23)) : (uint32_t)(D << (23 - p));
  const float hi = ff_bitsf(((uint32_t)fe << 23) | (mh & 0x7fffffu));
  float lo = 0.0f;
  if (p > 23) {
    const uint64_t r = D & ((1ull << (p - 23)) - 1);       // bits below hi's last place
    if (r) {
      const uint32_t rh = (uint32_t)(r >> 32), rl = (uint32_t)r;
      const int q = rh ? 63 - ff_clz(rh) : 31 - ff_clz(rl);
      const int ge = q + e2 + 127;
      if (ge >= 1) {
        const uint32_t ml = q >= 23 ? (uint32_t)(r >> (q - 23)) : (uint32_t)(r << (23 - q));
        lo = ff_bitsf(((uint32_t)ge << 23) | (ml & 0x7fffffu));
      }
    }
  }
  return ff_make(hi, lo);
}

// 1 - x for 0 <= x <= 1, with integer operations only.  For x in [0.5, 1) the double
// difference is exact (x = M 2^-53, 1 - x = (2^53 - M) 2^-53) and so is this pair up to its
// 48 bits: the relative accuracy of 1 - x holds as x -> 1.
FF_FN ff ff_one_minus_double_int(double x) {
  const uint64_t b = ff_dbits(x);
  if (((b >> 52) & 0x7ff) == 1022) {
    const uint64_t M = (b & 0xfffffffffffffull) | (1ull << 52);
    const uint64_t D = (1ull << 53) - M;
    return ff_from_mantissa(D, -53);
  }
  const ff xf = ff_from_double_int(x);
  const ff s = two_sum(1.0f, -xf.hi);
  return fast_two_sum(s.hi, f_sub(s.lo, xf.lo));
}

// A float as a double with integer operations: exact (infinities and NaN too), but 0 for zeros of
// either sign and below 2^-126.  Times 2^e for a finite f, e2 = e 2^20.
FF_FN double ff_widen(float f, int e2 = 0) {
  const uint32_t b = ff_fbits(f), m = b & 0x7fffffffu;
  if (m < 0x00800000u) return 0.0;
  const uint32_t h = ((m >> 3) + (0x38000000u + (uint32_t)e2)) | (m >= 0x7f800000u ? 0x7ff00000u : 0u);
  return ff_bitsd((uint64_t)((b & 0x80000000u) | h) << 32 | (uint32_t)(b << 29));
}
// hi + lo as a double, normalized or not.  A float-to-double conversion holds the FP64 pipe as long
// as an addition does, and what a walk waited on was that pipe: with the two conversions of a
// value in integers and the addition left, 1e6 tt events went from 304 to 267 us, 4.5e5 WW events
// from 88 to 73, 2^24 events over 64 channels from 1.62 to 1.55 ms and 5e5 tt events with their own
// beams from 238 to 221 us (there the addition was in integers as well, behind a normalization:
// for uniform beams that gave 302).
FF_FN double ff_to_double_int(ff a) { return ff_widen(a.hi) + ff_widen(a.lo); }

// f 2^e with f's high part put back into [1, 2), for |f| < 2^127: a product of many factors that
// stays in the floats' range whatever their sizes.  e counts in units of `unit`.
FF_FN void ff_renorm(ff &f, int &e, int unit) {
  const uint32_t b = ff_fbits(f.hi) & 0x7f800000u;
  const float scale = ff_bitsf(0x7f000000u - b);   // 2^(127 - exponent field), exact on both parts
  f = ff_make(f_mul(f.hi, scale), f_mul(f.lo, scale));
  e += ((int)(b >> 23) - 127) * unit;
}
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
inline
#endif
double ff_rare_ldexp(double d, int e) { return ldexp(d, e); }
// f 2^e as a double (finite f; the exponent goes into the widened parts, which then stay normal).
FF_FN double ff_to_double_scaled(ff f, int e) {
  if (e < -800 || e > 800) return ff_rare_ldexp(ff_to_double_int(f), e);
  return ff_widen(f.hi, e * 1048576) + ff_widen(f.lo, e * 1048576);
}

// ------------------------------------------------------------------ elementary functions
// Cody-Waite splits (three floats summing to the constant to ~2^-72 relative).
#define FF_PI128_1 0.024543693289160729f
#define FF_PI128_2 -6.8299044198028015e-10f
#define FF_PI128_3 -2.6798820468841905e-17f
#define FF_SIXTH_LO -4.9670538793122887e-09f  // 1/6 - (float)(1/6)
#define FF_LN2_32_1 0.021660849452018738f
#define FF_LN2_32_2 -5.9520444128935424e-11f
#define FF_LN2_32_3 -2.7447449183091686e-18f
#define FF_INV_PI128 40.743663787841797f    // 128/pi, for choosing the table index only
#define FF_INV_LN2_32 46.166240692138672f   // 32/ln 2, likewise
#define FF_PI_HI 3.1415927410125732f
#define FF_PI_LO -8.7422776573475858e-08f

// Tables (built per block in shared memory, fill_ff_tables in phs_kernels_ff.cu; on the host,
// ff_fill_tables):
//   trig[k] = {sin(k pi/128).hi, .lo, cos(k pi/128).hi, .lo}, k = 0..255
//   exp2[j] = {2^(j/32).hi, .lo}, j = 0..31
struct FFTables {
  float4 trig[256];
  float2 exp2[32];
};

// sin and cos of k pi/128 + f for |f| <= pi/256 (radians): sin f = f - f^3/6 + f^5/120 (the
// cubic term as a pair: tan next to 0 and cot next to pi/2 keep their relative accuracy) and
// q = 1 - cos f = f^2/2 - f^4/24 + f^6/720; terms below 2^-27 of the result run in float.  Then
// s_k + (c_k sin f - s_k q) and c_k - (s_k sin f + c_k q), where the parenthesis is below 2^-6.
// (80 instructions; a table of 64 entries, with a longer series in pairs, took 120.)
FF_FN void ff_sincos_table(int k, ff f, const FFTables &T, ff &s, ff &c) {
  const ff f2 = two_prod(f.hi, f.hi);
  const float f2lo = f_fma(f_add(f.hi, f.hi), f.lo, f2.lo);
  // g = f^2/6 - f^4/120, sin f = f - f g
  const float gh = f_mul(f2.hi, 1.0f / 6.0f);
  float gl = f_fma(f2.hi, 1.0f / 6.0f, -gh);
  gl = f_fma(f2.hi, FF_SIXTH_LO, f_fma(f2lo, 1.0f / 6.0f, gl));
  gl = f_fma(f_mul(f2.hi, f2.hi), -1.0f / 120.0f, gl);
  const float th = f_mul(f.hi, gh);
  const float tl = f_fma(f.lo, gh, f_fma(f.hi, gl, f_fma(f.hi, gh, -th)));
  const ff s1 = fast_two_sum(f.hi, -th);
  const ff sf = fast_two_sum(s1.hi, f_add(s1.lo, f_sub(f.lo, tl)));
  const float quart = f_mul(f_mul(f2.hi, f2.hi), f_fma(f2.hi, 1.0f / 720.0f, -1.0f / 24.0f));
  const ff q = ff_make(f_mul(f2.hi, 0.5f), f_fma(f2lo, 0.5f, quart));
  const float4 t = T.trig[k & 255];
  const ff sk = ff_make(t.x, t.y), ck = ff_make(t.z, t.w);
  s = ff_add(sk, ff_dot2_raw(ck, sf, ff_neg(sk), q));
  c = ff_sub(ck, ff_dot2_raw(sk, sf, ck, q));
}

// sin(2 pi x), cos(2 pi x) for x in [0, 1]: the reduction 256x - k is exact.
FF_FN void ff_sincos2pi(ff x, const FFTables &T, ff &s, ff &c) {
  const ff y = ff_make(f_mul(x.hi, 256.0f), f_mul(x.lo, 256.0f));
  const float kf = rintf(y.hi);
  const ff g = fast_two_sum(f_sub(y.hi, kf), y.lo);   // |g| <= 1/2; y.lo is below an ulp of y.hi
  ff_sincos_table((int)kf, ff_mul(g, ff_make(FF_PI128_1, FF_PI128_2)), T, s, c);
}

// sin and cos of z (radians), |z| <= pi/2 + pi/64: Cody-Waite reduction by k pi/128.
FF_FN void ff_sincos(ff z, const FFTables &T, ff &s, ff &c) {
  const float kf = rintf(f_mul(z.hi, FF_INV_PI128));
  ff f = ff_sub(z, two_prod(kf, FF_PI128_1));
  f = ff_add_f(f, f_mul(-kf, FF_PI128_2));
  f = ff_make(f.hi, f_fma(-kf, FF_PI128_3, f.lo));
  ff_sincos_table((int)kf, f, T, s, c);
}

// tan(z) for |z| < pi/2 (radians).
FF_FN ff ff_tan(ff z, const FFTables &T) {
  ff s, c;
  ff_sincos(z, T, s, c);
  return ff_div_fast(s, c);
}

// exp(y), |y| < 80.
FF_FN ff ff_exp(ff y, const FFTables &T) {
  float nf = rintf(f_mul(y.hi, FF_INV_LN2_32));
  ff r = ff_sub(y, two_prod(nf, FF_LN2_32_1));
  r = ff_add_f(r, f_mul(-nf, FF_LN2_32_2));
  r = ff_add_f(r, f_mul(-nf, FF_LN2_32_3));        // |r| <= ln2/64
  ff r2 = ff_sqr(r);
  float rh = r.hi;
  // exp r = 1 + r + r^2/2 + r^2 (r/6 + r^2/24 + r^3/120 + r^4/720)
  float tail = f_mul(r2.hi, f_mul(rh, f_fma(rh, f_fma(rh, f_fma(rh, 1.0f / 720.0f, 1.0f / 120.0f), 1.0f / 24.0f), 1.0f / 6.0f)));
  ff e = ff_add(ff_add_f(r, 1.0f), ff_mul_f(r2, 0.5f));
  e = ff_add_f(e, tail);
  int n = (int)nf;
  int j = n & 31, m = (n - j) / 32;
  float2 t = T.exp2[j];
  e = ff_mul(e, ff_make(t.x, t.y));
  float sc = ldexpf(1.0f, m);
  return ff_make(f_mul(e.hi, sc), f_mul(e.lo, sc));
}

// Fills the tables (host side).  Entries whose angle is a multiple of pi/2 are set to the
// exact 0 / +-1, so that tan near +-pi/2 keeps its relative accuracy.
inline void ff_fill_tables(FFTables &T) {
  for (int k = 0; k < 256; k++) {
    long double a = (long double)k * 3.14159265358979323846264338327950288L / 128.0L;
    long double sv = sinl(a), cv = cosl(a);
    if (k % 64 == 0) {
      sv = (k == 64) ? 1.0L : (k == 192 ? -1.0L : 0.0L);
      cv = (k == 0) ? 1.0L : (k == 128 ? -1.0L : 0.0L);
    }
    float sh = (float)sv, ch = (float)cv;
    T.trig[k].x = sh;
    T.trig[k].y = (float)(sv - (long double)sh);
    T.trig[k].z = ch;
    T.trig[k].w = (float)(cv - (long double)ch);
  }
  for (int j = 0; j < 32; j++) {
    long double v = exp2l((long double)j / 32.0L);
    float h = (float)v;
    T.exp2[j].x = h;
    T.exp2[j].y = (float)(v - (long double)h);
  }
}
