// phs_fix.h -- FP64 functions evaluated beside the FP64 pipe (host and device).
//
// GB300 issues a warp's FP64 instruction over 16 cycles of an SM (two lanes a cycle); a
// 32 x 32 -> 64 bit multiply-add takes 1.4, a 64 x 64 -> high 64 bit product 4.3 (measured).
// The functions here therefore run on the integer and FP32 pipes:
//
//   * square root and reciprocal: the seed 1/sqrt(x) or 1/x to about 2^-45 from the FP32
//     estimate and one Newton step in FP32 with the residual of the 48-bit operand, put
//     together as a double with integer operations; then one Newton step in FP64 with the
//     residual exact through the FMA (Markstein): 3 and 2 FP64 instructions;
//   * sin and cos of 2 pi x, tan, exp: 64-bit fixed point.  The argument is reduced exactly
//     (as integers), the Taylor series run in Horner form on 64-bit products, on 32-bit
//     ones where a term's weight is below 2^-29, and the result has about 2^-60 of
//     error before it is rounded to double.
//
// SM-cycles per call of a warp, measured with every warp in the same function (this header /
// the CUDA library): square root 55 / 152, reciprocal 38 / 92 (__drcp_rn), tan 127 / 622,
// exp 82 / 301, sin and cos of 2 pi x 122 with the conversion to double / 497 (sincospi).
// Beside FP64 work of other warps most of it is free.
//
// The header also compiles as host C++ (tests/test_fix_host.py checks the bounds stated).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define FX_FN __host__ __device__ __forceinline__
#else
#define FX_FN inline
#endif

// FP64 sums and products alone, with the same bits: a b = fma(a, b, -0), a + b = fma(a, 1, b).
// A fused multiply-add whose operands all sit in registers takes an SM's FP64 pipe 16 cycles a
// warp; a plain product or sum, and an FMA with a constant operand, 19 (measured, at any
// occupancy).  The two constants therefore live in registers: the caller reads them once per
// thread from memory (fx_regs), where the compiler cannot see their values.
struct FxRegs {
  double nz, one;   // -0.0 and 1.0
};
#if defined(__CUDACC__)
namespace {
__constant__ double fx_reg_values[4] = {-0.0, 1.0, -0.0, 1.0};
}
// Per thread (not warp-uniform to the compiler, which would keep them as constant operands).
__device__ __forceinline__ FxRegs fx_regs() {
  const int i = (threadIdx.x & 1) * 2;
  return {fx_reg_values[i], fx_reg_values[i + 1]};
}
#endif

#if defined(__CUDA_ARCH__)
FX_FN uint64_t fx_mulhi(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
FX_FN uint32_t fx_mulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
FX_FN int fx_clz64(uint64_t a) { return __clzll((long long)a); }
FX_FN uint32_t fx_hi(double d) { return (uint32_t)__double2hiint(d); }
FX_FN uint32_t fx_lo(double d) { return (uint32_t)__double2loint(d); }
FX_FN double fx_double(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
FX_FN uint64_t fx_bits(double d) { return (uint64_t)__double_as_longlong(d); }
FX_FN double fx_from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
FX_FN float fx_float(uint32_t b) { return __uint_as_float(b); }
FX_FN uint32_t fx_fbits(float f) { return __float_as_uint(f); }
FX_FN float fx_rsqrt_est(float a) { return rsqrtf(a); }
FX_FN float fx_rcp_est(float a) { return __fdividef(1.0f, a); }
FX_FN float fx_fmaf(float a, float b, float c) { return __fmaf_rn(a, b, c); }
FX_FN float fx_mulf(float a, float b) { return __fmul_rn(a, b); }
FX_FN float fx_minf(float a, float b) { return fminf(a, b); }
FX_FN float fx_maxf(float a, float b) { return fmaxf(a, b); }
FX_FN int fx_rint32(float a) { return __float2int_rn(a); }
FX_FN uint32_t fx_trunc_u32(float a) { return __float2uint_rz(a); }
FX_FN double fx_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
FX_FN uint64_t fx_mulhi(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
FX_FN uint32_t fx_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
FX_FN int fx_clz64(uint64_t a) { return a ? __builtin_clzll(a) : 64; }
FX_FN uint64_t fx_bits(double d) { uint64_t b; memcpy(&b, &d, 8); return b; }
FX_FN double fx_from_bits(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
FX_FN uint32_t fx_hi(double d) { return (uint32_t)(fx_bits(d) >> 32); }
FX_FN uint32_t fx_lo(double d) { return (uint32_t)fx_bits(d); }
FX_FN double fx_double(uint32_t hi, uint32_t lo) { return fx_from_bits((uint64_t)hi << 32 | lo); }
FX_FN float fx_float(uint32_t b) { float f; memcpy(&f, &b, 4); return f; }
FX_FN uint32_t fx_fbits(float f) { uint32_t b; memcpy(&b, &f, 4); return b; }
FX_FN float fx_rsqrt_est(float a) { return 1.0f / sqrtf(a); }
FX_FN float fx_rcp_est(float a) { return 1.0f / a; }
FX_FN float fx_fmaf(float a, float b, float c) { return fmaf(a, b, c); }
FX_FN float fx_mulf(float a, float b) { return a * b; }
FX_FN float fx_minf(float a, float b) { return a < b ? a : b; }
FX_FN float fx_maxf(float a, float b) { return a > b ? a : b; }
FX_FN int fx_rint32(float a) { return (int)lrintf(a); }
FX_FN uint32_t fx_trunc_u32(float a) { return (uint32_t)a; }
FX_FN double fx_fma(double a, double b, double c) { return fma(a, b, c); }
#endif

FX_FN double fx_mul(const FxRegs &k, double a, double b) { return fx_fma(a, b, k.nz); }
FX_FN double fx_add(const FxRegs &k, double a, double b) { return fx_fma(a, k.one, b); }
FX_FN double fx_sub(const FxRegs &k, double a, double b) { return fx_fma(-b, k.one, a); }
FX_FN double fx_neg(double a) { return fx_double(fx_hi(a) ^ 0x80000000u, fx_lo(a)); }
// a 2^e for a normal result (zeros, subnormals, infinities and NaN come back unchanged).
FX_FN double fx_scale(double a, int e) {
  const uint32_t h = fx_hi(a);
  return (h & 0x7ff00000u) - 0x00300000u < 0x7f900000u ? fx_double(h + (uint32_t)(e << 20), fx_lo(a)) : a;
}

// The library's functions for the arguments that the forms here leave out.  On the device they
// are calls: inlined at every use they would be most of the kernels' code, and the walks'
// instruction fetches already limit them.
#if defined(__CUDACC__)
#define FX_RARE static __host__ __device__ __noinline__
#else
#define FX_RARE inline
#endif
FX_RARE double fx_lib_sqrt(double x) { return sqrt(x); }
FX_RARE double fx_lib_div(double a, double b) { return a / b; }
FX_RARE double fx_lib_exp(double x) { return exp(x); }
FX_RARE double fx_lib_log(double x) { return log(x); }
FX_RARE double fx_lib_atan2(double y, double x) { return atan2(y, x); }
FX_RARE double fx_lib_sin(double x) { return sin(x); }
FX_RARE double fx_lib_cos(double x) { return cos(x); }

// ------------------------------------------------------------ square root and reciprocal
// y0 + c (y0 in [0.5, 1), |c| < 2^-21) as a double: y0's bits widened, c added in units of twice
// its last place.  (With an estimate 2 ulps off and the operand's low bits |c| reaches 1.1 2^-22.
// The callers clamp their estimates to [0.5, 1): the true value lies there, but an estimate within
// its 2 ulps may not, and in the binade below c would count half.)
FX_FN uint64_t fx_seed(float y0, float c) {
  const uint32_t b = fx_fbits(y0);
  const uint64_t d = (uint64_t)((b >> 3) + ((1023u - 127u) << 20)) << 32 | (uint64_t)(b << 29);
  return d + 2 * (uint64_t)(int64_t)fx_rint32(fx_mulf(c, 0x1p52f));
}

// 1/sqrt(x) to about 2^-45 for a normal x > 0; the bits of a double.
FX_FN uint64_t fx_rsqrt_seed(double x) {
  const uint32_t hi = fx_hi(x), lo = fx_lo(x);
  const uint32_t be = hi >> 20, even = (be & 1u) ^ 1u;   // x = m 4^j, m in [1, 4)
  const float mh = fx_float(((127u + even) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const float ml = fx_mulf((float)(lo & 0x1fffffffu), even ? 0x1p-51f : 0x1p-52f);
  float y0 = fx_rsqrt_est(mh);
  y0 = fx_minf(fx_maxf(y0, 0.5f), 0x1.fffffep-1f);
  const float p = fx_mulf(y0, y0), pl = fx_fmaf(y0, y0, -p);
  float e = fx_fmaf(-mh, p, 1.0f);             // 1 - m y0^2
  e = fx_fmaf(-mh, pl, e);
  e = fx_fmaf(-ml, p, e);
  const float c = fx_mulf(fx_mulf(y0, e), fx_fmaf(e, 0.375f, 0.5f));
  const int j = ((int)be - 1023) >> 1;
  return fx_seed(y0, c) - ((uint64_t)(int64_t)j << 52);
}

// sqrt(x): the correctly rounded value but for arguments whose root lies within 2^-30 ulp
// of a rounding boundary.  Zeros, subnormals and the smallest normals (whose residual would
// be subnormal), infinities and NaN go to the library's; negatives give NaN.
FX_FN double fx_sqrt(double x, const FxRegs &k = FxRegs{-0.0, 1.0}) {
  const uint32_t hi = fx_hi(x);
  if (hi - 0x08000000u >= 0x77f00000u) {
    if (hi > 0x80000000u) return fx_double(0x7fffffffu, 0xffffffffu);   // negative
    return fx_lib_sqrt(x);
  }
  const uint64_t rb = fx_rsqrt_seed(x);
  const double r = fx_from_bits(rb), h = fx_from_bits(rb - (1ull << 52));
  const double s = fx_mul(k, x, r);
  return fx_fma(fx_fma(-s, s, x), h, s);
}

// 1/x within an ulp (almost always correctly rounded) for x > 0.
FX_FN double fx_rcp(double x, const FxRegs &k = FxRegs{-0.0, 1.0}) {
  const uint32_t hi = fx_hi(x), lo = fx_lo(x);
  if (hi - 0x04000000u >= 0x78000000u) return fx_lib_div(1.0, x);
  const float mh = fx_float((127u << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const float ml = fx_mulf((float)(lo & 0x1fffffffu), 0x1p-52f);
  float y0 = fx_rcp_est(mh);
  y0 = fx_minf(fx_maxf(y0, 0.5f), 0x1.fffffep-1f);
  float e = fx_fmaf(-mh, y0, 1.0f);
  e = fx_fmaf(-ml, y0, e);
  const float c = fx_mulf(y0, fx_fmaf(e, e, e));
  const double r = fx_from_bits(fx_seed(y0, c) - ((uint64_t)(int64_t)((int)(hi >> 20) - 1023) << 52));
  return fx_fma(fx_fma(-x, r, k.one), r, r);
}

// a / b given r = fx_rcp(b): the product corrected once with its residual, the correctly rounded
// quotient (Markstein) where r is 1/b correctly rounded, as it is but for about one b in 2^36,
// and the residual is not subnormal.
FX_FN double fx_quot(double a, double b, double r, const FxRegs &k) {
  const double q = fx_mul(k, a, r);
  return fx_fma(fx_fma(-q, b, a), r, q);
}
// b and a such that fx_quot serves a / b: b normal, positive, neither huge nor tiny; a neither
// huge nor infinite (the residual of an infinite quotient is no number).
FX_FN bool fx_quot_serves(double b) { return fx_hi(b) - 0x20b00000u < 0x3e800000u; }   // 2^-500 .. 2^500
FX_FN bool fx_quot_serves(double a, double b) {
  return fx_quot_serves(b) && (fx_hi(a) & 0x7fffffffu) < 0x5f300000u;
}
FX_FN double fx_div(double a, double b, const FxRegs &k) {
  if (!fx_quot_serves(a, b)) return fx_lib_div(a, b);
  return fx_quot(a, b, fx_rcp(b, k), k);
}

// a > b; as integers where neither is negative or NaN.
FX_FN bool fx_gt(double a, double b) {
  const uint32_t ah = fx_hi(a), bh = fx_hi(b);
  if ((ah > bh ? ah : bh) <= 0x7fefffffu) return fx_bits(a) > fx_bits(b);
  return a > b;
}

// ---------------------------------------------------------------------- packing
// m 2^e (m > 0 an integer) as a double, rounded to nearest; e such that the result is normal.
FX_FN double fx_pack(uint64_t m, int e) {
  const int z = fx_clz64(m);
  m <<= z;
  // bit 63 of m lands on the exponent field's lowest bit: one less is put there
  const uint64_t r = (m >> 11) + ((m >> 10) & 1u);
  return fx_from_bits(r + ((uint64_t)(uint32_t)(e - z + 63 + 1022) << 52));
}

// A value of Q62 (v 2^-62) as a double.
FX_FN double fx_from_q62(int64_t v) {
  const uint64_t a = v < 0 ? (uint64_t)-v : (uint64_t)v;
  if (a == 0) return 0.0;
  const double d = fx_pack(a, -62);
  return v < 0 ? fx_neg(d) : d;
}

// x 2^64 for 0 <= x < 1, truncated to an integer (exact for x >= 2^-11).
FX_FN uint64_t fx_q64(double x) {
  const uint64_t b = fx_bits(x);
  const int be = (int)(b >> 52);
  const uint64_t m = (b << 11) | (1ull << 63);
  const int sh = 1022 - be;                     // >= 0
  return sh < 64 ? m >> sh : 0;
}

// ---------------------------------------------------------------------- sin, cos, tan
// For v = u^2 (Q64), 0 <= u <= pi/4: w = 1 - sin(u)/u and k = 1 - cos(u), both Q64, by
// their Taylor series in Horner form (the next terms are below 2^-63 and 2^-68).  Terms of
// weight below 2^-28 run on 32-bit products; together within 2^-59.
FX_FN void fx_sincos_series(uint64_t v, uint64_t &w, uint64_t &k) {
  const uint32_t vh = (uint32_t)(v >> 32);
  // 1/11! - v (1/13! - v (1/15! - v / 17!)), Q57, and 1/12! - v (1/14! - v (1/16! - v / 18!)), Q60
  uint32_t a = 0x1ae7fu - fx_mulhi32(vh, 0x195u);
  uint32_t b = 0xd740u - fx_mulhi32(vh, 0xb4u);
  a = 0x1612461u - fx_mulhi32(vh, a);
  b = 0xc9cba5u - fx_mulhi32(vh, b);
  a = 0xd7322b40u - fx_mulhi32(vh, a);
  b = 0x8f76c780u - fx_mulhi32(vh, b);
  uint64_t s = 0x2e3bc74aad8eull - (((uint64_t)vh * a) >> 25);   // 1/9! - v (...), Q64
  uint64_t c = 0x49f93edde28ull - (((uint64_t)vh * b) >> 28);   // 1/10! - v (...)
  s = 0xd00d00d00d00dull - fx_mulhi(v, s);                        // 1/7!
  c = 0x1a01a01a01a02ull - fx_mulhi(v, c);                        // 1/8!
  s = 0x222222222222222ull - fx_mulhi(v, s);                      // 1/5!
  c = 0x5b05b05b05b05bull - fx_mulhi(v, c);                      // 1/6!
  s = 0x2aaaaaaaaaaaaaabull - fx_mulhi(v, s);                      // 1/3!
  c = 0xaaaaaaaaaaaaaabull - fx_mulhi(v, c);                      // 1/4!
  c = 0x8000000000000000ull - fx_mulhi(v, c);                     // 1/2!
  w = fx_mulhi(v, s);
  k = fx_mulhi(v, c);
}

// sin and cos of 2 pi x for 0 <= x < 1 given as X = x 2^64, Q62, within 2^-58.
FX_FN void fx_sincos2pi_q62(uint64_t X, int64_t &s, int64_t &c) {
  const uint32_t q = (uint32_t)((X + (1ull << 61)) >> 62);        // nearest quarter turn, mod 4
  const int64_t r = (int64_t)(X - ((uint64_t)q << 62));           // |r| <= 2^61
  uint64_t ar = r < 0 ? (uint64_t)-r : (uint64_t)r;
  ar -= ar >> 61;                                                 // an odd eighth: below 2^61
  const uint64_t u = fx_mulhi(ar << 3, 0xc90fdaa22168c235ull);    // 2 pi r 2^-64, Q64
  uint64_t w, k;
  fx_sincos_series(fx_mulhi(u, u), w, k);
  int64_t sn = (int64_t)((u - fx_mulhi(u, w)) >> 2);
  const int64_t cs = (int64_t)((1ull << 62) - (k >> 2));
  sn = r < 0 ? -sn : sn;
  // quarter turns: (s, c) -> (c, -s) -> (-s, -c) -> (-c, s)
  const int64_t a = q & 1u ? cs : sn, b = q & 1u ? sn : cs;
  s = q & 2u ? -a : a;
  c = ((q + 1u) & 2u) ? -b : b;
}

// sin of the angle un 2^(-61 - z) below 2^-9, un normalized (0, or within a factor 4 of 2^64):
// within 0.52 ulp of itself.  (A call: one angle in 500 needs it, and always normalizing the residual
// took 1e7 tt events from 5180 to 5390 us.)
FX_RARE double fx_sin_small(uint64_t un, int z) {
  const uint64_t u = z < 67 ? un >> (z - 3) : 0;                  // Q64
  const uint64_t v = fx_mulhi(u, u);
  // 1 - sin(u) / u = v (1/3! - v (1/5! - ..)), Q64
  const uint64_t sn = un - fx_mulhi(un, fx_mulhi(v, 0x2aaaaaaaaaaaaaabull - fx_mulhi(v, 0x222222222222222ull - fx_mulhi(v, 0xd00d00d00d00dull))));
  return sn == 0 ? 0.0 : fx_pack(sn, -61 - z);
}
// The sine or cosine that is small at q quarter turns and +-angle, where sin(angle) = small.
FX_FN void fx_put_small(double small, uint32_t q, bool minus, double &s, double &c) {
  const bool odd = q & 1u;
  if (small != 0.0 && (minus != ((odd ? q + 1u : q) & 2u ? true : false))) small = fx_neg(small);
  s = odd ? s : small;
  c = odd ? small : c;
}
// sin and cos of 2 pi x for 0 <= x < 1: in Q62, and again below 2^-9 (there from x's own bits, which
// x 2^64 truncates, or from the residual, which is exact): within 1.2 ulp of themselves.
FX_FN void fx_sincos2pi(double x, double &s, double &c) {
  const uint64_t X = fx_q64(x);
  int64_t si, ci;
  fx_sincos2pi_q62(X, si, ci);
  s = fx_from_q62(si);
  c = fx_from_q62(ci);
  const uint32_t q = (uint32_t)((X + (1ull << 61)) >> 62);
  const int64_t r = (int64_t)(X - ((uint64_t)q << 62));
  const uint64_t ar = r < 0 ? (uint64_t)-r : (uint64_t)r;
  if (ar < 1ull << 52) {
    const uint32_t hi = fx_hi(x);
    int z = fx_clz64(ar);
    uint64_t un = z < 64 ? ar << z : 0;                           // un 2^(-64 - z) turns
    if (hi < 0x3fc00000u) {
      z = 1022 - (int)(hi >> 20);
      un = hi < 0x00100000u ? 0 : (fx_bits(x) << 11) | (1ull << 63);
    }
    fx_put_small(fx_sin_small(fx_mulhi(un, 0xc90fdaa22168c235ull), z), q, r < 0, s, c);
  }
}

// 2^126 / d for d in [2^62, 2^64), to 2^-43.
FX_FN uint64_t fx_recip_q62(uint64_t d) {
  const float y0 = fx_rcp_est((float)(uint32_t)(d >> 32));        // in [2^-32, 2^-30]
  const uint32_t Y0 = fx_trunc_u32(fx_mulf(y0, 0x1.fffffcp+61f)); // 2^94 / d to 2^-22, below it
  // 1 - d Y0 2^-94, in units of 2^-62
  const uint32_t dh = (uint32_t)(d >> 32), dl = (uint32_t)d;
  const int64_t e = (int64_t)((1ull << 62) - ((uint64_t)dh * Y0 + (((uint64_t)dl * Y0) >> 32)));
  return ((uint64_t)Y0 << 32) + (uint64_t)(((int64_t)(int32_t)(e >> 12) * (int64_t)(Y0 >> 1)) >> 17);
}

// n / d for n, d in [2^62, 2^64): the quotient in Q62, within 2^-60 of it.
FX_FN uint64_t fx_div_q62(uint64_t n, uint64_t d) {
  const uint64_t Y = fx_recip_q62(d);
  const uint64_t q = fx_mulhi(n, Y);                              // n / d, Q62, to 2^-43
  const int32_t r = (int32_t)(int64_t)((n >> 2) - fx_mulhi(q, d)); // its residual, 2^-62 d
  return q + (uint64_t)(((int64_t)r * (int64_t)(uint32_t)(Y >> 33)) >> 29);
}

// tan(z) for |z| < pi/2 as doubles: within 0.51 ulp.  z and, above pi/4, pi/2 - |z| are reduced
// exactly and stay normalized.
FX_FN double fx_tan(double z) {
  const uint32_t zh = fx_hi(z);
  const int be = (int)((zh >> 20) & 0x7ffu);                      // <= 1023
  const uint64_t mn = (fx_bits(z) << 11) | (1ull << 63);          // |z| = mn 2^(be - 1086)
  const uint64_t A = 1023 - be < 64 ? mn >> (1023 - be) : 0;      // |z|, Q63
  uint64_t un = mn;                                               // u = un 2^(e - 63)
  int e = be - 1023;
  const bool big = A > 0x6487ed5110b4611aull;                     // above pi/4: u = pi/2 - |z|
  if (big) {
    const uint64_t d = 0xc90fdaa22168c234ull - A;                 // > 0: |z| below pi/2
    const int sh = fx_clz64(d);
    un = (d << sh) | ((0xc4c6628b80dc1cd1ull >> 1) >> (63 - sh));
    e = -sh;
  }
  const uint64_t u = -1 - e < 64 ? un >> (-1 - e) : 0;            // Q64
  uint64_t w, k;
  fx_sincos_series(fx_mulhi(u, u), w, k);
  const uint64_t sn = un - fx_mulhi(un, w);                       // sin u = sn 2^(e - 63)
  const uint64_t cs = (1ull << 63) - (k >> 1);                    // cos u, Q63
  const uint64_t q = fx_div_q62(big ? cs : sn, big ? sn : cs);
  const double t = fx_pack(q, (big ? -e : e) - 62);
  return (int32_t)zh < 0 ? fx_neg(t) : t;
}

// ---------------------------------------------------------------------- exp
// exp(y): for 0 <= y < 708 in fixed point (2^n 2^(j/4) exp(u), u < ln(2)/4, Taylor terms
// through u^12) within 0.51 ulp, else the library's.
FX_FN double fx_exp(double y) {
  const uint32_t yh = fx_hi(y);
  if (yh >= 0x40862000u) return fx_lib_exp(y);
  const int sh = 1085 - (int)(yh >> 20);                          // >= 53
  const uint64_t mn = (fx_bits(y) << 11) | (1ull << 63);
  const uint64_t L = 0xb8aa3b295c17f0bcull;                       // log2(e), Q63
  const uint64_t ph = fx_mulhi(mn, L), pl = mn * L;               // y log2(e) = ph 2^-sh
  const int n = sh < 64 ? (int)(ph >> sh) : 0;
  const uint64_t f = sh < 64 ? (ph << (64 - sh)) | (pl >> sh) : (sh < 128 ? ph >> (sh - 64) : 0);
  const uint32_t j = (uint32_t)(f >> 62);
  const uint64_t u = fx_mulhi(f & 0x3fffffffffffffffull, 0xb17217f7d1cf79acull);   // Q64
  const uint32_t uh = (uint32_t)(u >> 32);
  // 1/7! + u (1/8! + u (... + u / 12!)), Q44
  uint32_t a = 440721u + fx_mulhi32(uh, 36727u);
  a = 4847935u + fx_mulhi32(uh, a);
  a = 48479349u + fx_mulhi32(uh, a);
  a = 436314138u + fx_mulhi32(uh, a);
  a = 3490513104u + fx_mulhi32(uh, a);
  uint64_t t = 0x5b05b05b05b05bull + (((uint64_t)uh * a) >> 12);   // 1/6! + u (...), Q64
  t = 0x222222222222222ull + fx_mulhi(u, t);
  t = 0xaaaaaaaaaaaaaabull + fx_mulhi(u, t);
  t = 0x2aaaaaaaaaaaaaabull + fx_mulhi(u, t);
  t = 0x8000000000000000ull + fx_mulhi(u, t);
  t = 0x8000000000000000ull + (fx_mulhi(u, t) >> 1);    // 1 + u (1/2 + ...), Q63
  t = 0x8000000000000000ull + fx_mulhi(u, t);           // exp(u), Q63
  const uint64_t c = j & 2u ? (j & 1u ? 0xd744fccad69d6af4ull : 0xb504f333f9de6484ull)
                            : (j & 1u ? 0x9837f0518db8a96full : 0x8000000000000000ull);
  return fx_pack(fx_mulhi(t, c), n - 62);
}

// ---------------------------------------------------------------------- inverse functions
// sin and cos of phi (radians, 0 <= phi < 8): the phase in turns, then fx_sincos2pi_q62; within
// 2^-58, and correctly rounded like the library's but for about one value in a hundred; a small phi's
// sine within 0.52 ulp of itself.
FX_FN void fx_sincos(double phi, double &s, double &c) {
  const uint32_t hi = fx_hi(phi);
  if (hi >= 0x40200000u) {   // 8 and above, negative, NaN
    s = fx_lib_sin(phi);
    c = fx_lib_cos(phi);
    return;
  }
  const uint64_t mn = (fx_bits(phi) << 11) | (1ull << 63);        // phi = mn 2^(be - 1086)
  const int sh = 1024 - (int)(hi >> 20);                          // >= -1
  const uint64_t C = 0xa2f9836e4e44152aull;                       // 2^66 / (2 pi)
  const uint64_t ph = fx_mulhi(mn, C), pl = mn * C;               // phi 2^64 / (2 pi) = ph 2^-sh
  const uint64_t X = sh < 0 ? (ph << 1) | (pl >> 63) : (sh < 64 ? ph >> sh : 0);
  int64_t si, ci;
  fx_sincos2pi_q62(X, si, ci);
  s = fx_from_q62(si);
  c = fx_from_q62(ci);
  if (hi < 0x3f600000u) s = hi < 0x00100000u ? 0.0 : fx_sin_small(mn, sh + 1);   // below 2^-9
}

// atan2(y, x) for finite arguments whose exponents lie within 2^+-400 (others: the library's).
// With t the smaller over the larger magnitude: below 2^-9 the series of atan(t) in FP64;
// else an FP32 estimate u of atan(t) and the remaining angle, tan(d) = (lo cos u - hi sin u) /
// (hi cos u + lo sin u), in fixed point (|d| < 2^-20, so d^3/3 is below 2^-61 of it).  Within
// 0.51 ulp above 2^-4 and an ulp everywhere.
FX_FN double fx_atan2(double y, double x) {
  const uint32_t yh = fx_hi(y) & 0x7fffffffu, xh = fx_hi(x) & 0x7fffffffu;
  if (yh - 0x26f00000u >= 0x32000000u || xh - 0x26f00000u >= 0x32000000u) return fx_lib_atan2(y, x);
  const uint64_t yb = fx_bits(y) & 0x7fffffffffffffffull, xb = fx_bits(x) & 0x7fffffffffffffffull;
  const bool swap = yb > xb, back = (int32_t)fx_hi(x) < 0;
  const uint64_t hb = swap ? yb : xb, lb = swap ? xb : yb;
  const int d = (int)(hb >> 52) - (int)(lb >> 52);                // >= 0
  uint64_t th;                                                    // atan(t), Q64
  double r;
  if (d > 9) {
    const double t = fx_from_bits(lb) / fx_from_bits(hb), t2 = t * t;
    r = t + t * t2 * (-1.0 / 3.0 + t2 * (0.2 + t2 * (-1.0 / 7.0 + t2 * (1.0 / 9.0))));
    const int sh = 1022 - (int)(fx_hi(r) >> 20);                  // r < 2^-8
    th = sh < 64 ? ((fx_bits(r) << 11) | (1ull << 63)) >> sh : 0;
  } else {
    const uint64_t H = (hb << 11) | (1ull << 63), L = ((lb << 11) | (1ull << 63)) >> d;   // Q63
    const float t = fx_mulf((float)(uint32_t)(L >> 32), fx_rcp_est((float)(uint32_t)(H >> 32)));
    const uint32_t u = fx_trunc_u32(fx_mulf(atanf(t), 0x1p32f));
    uint64_t w, k;
    fx_sincos_series((uint64_t)u * u, w, k);
    const uint64_t U = (uint64_t)u << 32;
    const uint64_t sn = U - fx_mulhi(U, w), cs = 0 - k;           // Q64 (t >= 2^-10: cos u < 1)
    // lo cos u - hi sin u, 2^-127 units, kept in 2^-82
    const uint64_t a1 = fx_mulhi(L, cs), a0 = L * cs;
    const uint64_t b1 = fx_mulhi(H, sn), b0 = H * sn;
    const uint64_t n0 = a0 - b0, n1 = a1 - b1 - (a0 < b0 ? 1 : 0);
    const int64_t N = (int64_t)((n1 << 19) | (n0 >> 45));
    const uint64_t Y = fx_recip_q62((fx_mulhi(H, cs) >> 1) + (fx_mulhi(L, sn) >> 1));   // 2^126 / (.)
    // N Y 2^-64, signed: tan(d) in 2^-82
    const uint64_t an = N < 0 ? (uint64_t)-N : (uint64_t)N;
    const uint64_t q = fx_mulhi(an, Y) >> 18;
    th = N < 0 ? U - q : U + q;
    r = fx_pack(th, -64);
  }
  if (swap || back) {
    uint64_t T = th >> 3;                                         // Q61
    if (swap) T = 0x3243f6a8885a308dull - T;                      // pi/2 - .
    if (back) T = 0x6487ed5110b4611aull - T;                      // pi - .
    r = fx_pack(T, -61);
  }
  return (int32_t)fx_hi(y) < 0 ? fx_neg(r) : r;
}

// log(v) for a normal v > 0 (others: the library's): m in [sqrt(1/2), sqrt(2)), s = (m - 1) /
// (m + 1), log m = 2 s (1 + s^2/3 + s^4/5 + ...) in fixed point with a relative error of 2^-59,
// and e log 2 added in FP64.  Within 0.51 ulp where e is 0, an ulp elsewhere.
FX_FN double fx_log(double v) {
  const uint32_t hi = fx_hi(v);
  if (hi - 0x00100000u >= 0x7fe00000u) return fx_lib_log(v);
  const uint64_t f = (fx_bits(v) << 11) | (1ull << 63);           // 1.f, Q63
  const bool up = f >= 0xb504f333f9de6484ull;                     // above sqrt(2): m = f / 2
  const int e = (int)(hi >> 20) - 1023 + (up ? 1 : 0);
  // |m - 1| and m + 1
  uint64_t n = up ? 0 - f : (f << 1) >> 1;                        // Q64 : Q63
  const uint64_t dn = (1ull << 62) + (f >> (up ? 2 : 1));         // Q62
  if (n == 0) return (double)e * 0x1.62e42fefa39efp-1;
  const int z = fx_clz64(n);
  n <<= z;
  const uint64_t q = fx_div_q62(n, dn);
  const int ex = (up ? 2 : 1) + z;                                // s = q 2^-62 2^-ex
  const uint64_t S = ex < 2 ? q << (2 - ex) : (ex < 66 ? q >> (ex - 2) : 0);    // Q64, below 0.172
  const uint64_t w = fx_mulhi(S, S);
  const uint32_t wh = (uint32_t)(w >> 32);
  uint32_t p = 0xb21642du + fx_mulhi32(wh, 0xa3d70a4u);           // 1/23 + w/25, Q32
  p = 0xc30c30cu + fx_mulhi32(wh, p);
  p = 0xd79435eu + fx_mulhi32(wh, p);
  p = 0xf0f0f0fu + fx_mulhi32(wh, p);
  p = 0x11111111u + fx_mulhi32(wh, p);
  p = 0x13b13b14u + fx_mulhi32(wh, p);
  uint64_t P = 0x1745d1745d1745d1ull + (uint64_t)wh * p;          // 1/11 + w (...), Q64
  P = 0x1c71c71c71c71c72ull + fx_mulhi(w, P);
  P = 0x2492492492492492ull + fx_mulhi(w, P);
  P = 0x3333333333333333ull + fx_mulhi(w, P);
  P = 0x5555555555555555ull + fx_mulhi(w, P);
  const uint64_t t = (1ull << 63) + (fx_mulhi(w, P) >> 1);        // 1 + w P, Q63
  const double lm = fx_pack(fx_mulhi(q, t), -60 - ex);       // 2 s t
  const double l = up ? fx_neg(lm) : lm;
  return e == 0 ? l : fx_fma((double)e, 0x1.62e42fefa39efp-1, fx_fma((double)e, 0x1.abc9e3b39803fp-56, l));
}
