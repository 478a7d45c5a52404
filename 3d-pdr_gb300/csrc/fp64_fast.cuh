// fp64_fast.cuh -- FP64 elementary functions for a GPU whose FP64 pipe is the
// scarce unit.
//
// On GB300 an FP64 warp instruction (DFMA, DADD, DMUL, a compare, a conversion
// to or from FP64) holds a sub-partition's FP64 pipe for 64 to 76 cycles
// whatever its active lanes; an FP32 FMA takes 1, an integer operation 1 to 2.
// Measured per warp and call: exp 1,216 cycles, log 2,220, pow 6,340, a
// division 548, sqrt 650.  The kernels that evaluate rates and escape
// probabilities do little else.  Here each function keeps in FP64 only the two
// or three operations that carry the leading bits; argument splitting,
// conversions and the high-order terms run on the integer and FP32 pipes:
//
//  * exponentials are 2^((k + r)/1024) with the integer k found in FP32, the
//    remainder r by one FMA, 2^(j/1024) from a table (Tang 1989) and a short
//    series; its terms beyond z^2/2 are below 5e-11 and evaluated in FP32;
//  * logarithms are 1024 log2(x) = h + l from a 512-row table of c ~ 1/m with
//    r = m c - 1 exact in one FMA;
//  * a small FP32 correction t of an FP64 coefficient c with a known exponent
//    is added as an integer to c's mantissa (add_rel), not by a conversion and
//    an FP64 add;
//  * divisions, reciprocals and square roots start from the FP32 unit's value
//    and are finished by FP64 residual steps (Markstein 2000).
//
// Against 113-bit references over the ranges the kernels use (3,000,000 points
// each, on the CPU): exp_fast 0.502 ulp, powk 0.70 ulp, log2k 1.5e-14 of
// 1024 log2(x) absolute, rsqrt_fast 0.64 ulp; div_fast rounds as the division
// in every one, and to 0.5 + 2^-35 ulp by its construction, as rcp_near.  sqrt_rn
// rounds as the IEEE square root for every operand.
#pragma once

#include <cuda_runtime.h>

namespace pdr {
namespace fp64 {

#include "fp64_tables.inc"
static_assert(alignof(ExpRow) == alignof(double2), "a row is read with one 16-byte load");
static_assert(alignof(LogRow) == alignof(float2), "c and lo of a row are read with one 8-byte load");

constexpr double K_LN2 = 1477.3197218702985;        // 1024/ln 2
constexpr float K_LN2_LO = 2.08438003e-14f;         //   its rounding error
constexpr double C1 = 0.00067690154351557157;       // ln 2/1024
constexpr double C2 = 2.2909784980688164e-07;       // C1^2/2 = 1.9218... 2^-23

#ifdef __CUDACC__   // (a host build of this file brings its own)
// the FP32 unit's approximations, to about an ulp
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
#endif

__device__ __forceinline__ int hi32(double x) { return __double2hiint(x); }
__device__ __forceinline__ int lo32(double x) { return __double2loint(x); }

// FP32 -> FP64, exact, for zero and normal values
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned mag = u & 0x7fffffffu;
  const unsigned h = (u & 0x80000000u) | (mag ? (mag >> 3) + 0x38000000u : 0u);
  return __hiloint2double((int)h, (int)(u << 29));
}
// FP64 -> FP32 by truncation; magnitudes below 2^-126 give zero, above 2^127 are not allowed
__device__ __forceinline__ float d2f(double x) {
  const unsigned h = (unsigned)hi32(x);
  const unsigned mag = h & 0x7fffffffu;
  const unsigned m = __funnelshift_l((unsigned)lo32(x), mag - 0x38000000u, 3);
  return __uint_as_float(mag < 0x38100000u ? 0u : ((h & 0x80000000u) | m));
}
// c (1 + t) for |t| < 2^-6, in integer arithmetic; mant = c's mantissa in [1, 2),
// which stays in its binade
__device__ __forceinline__ double add_rel(double c, float mant, float t) {
  const int n = __float2int_rn(t * (mant * 68719476736.0f));   // 2^36
  return __longlong_as_double(__double_as_longlong(c) + ((long long)n << 16));
}
__device__ __forceinline__ double flip(double x) { return __hiloint2double(hi32(x) ^ (int)0x80000000u, lo32(x)); }
// x 2^e for results in the normal range
__device__ __forceinline__ double scale2(double x, int e) { return __hiloint2double(hi32(x) + (e << 20), lo32(x)); }

// nearest integer of |x| < 2^22 in FP32
__device__ __forceinline__ int rint_f(float x, float &rounded) {
  const float t = x + 12582912.0f;
  rounded = t - 12582912.0f;
  return __float_as_int(t) - 0x4b400000;
}

// u with 2^(r/1024) = 1 + r u, |r| <= 2: C1 + r C2 (1 + z/3 + z^2/12 + ...), z = r C1
__device__ __forceinline__ double exp2_slope(double r) {
  const float rf = d2f(r);
  constexpr float A = (float)(C1 / 3.0), B = (float)(C1 * C1 / 12.0);
  const double c2 = add_rel(C2, 1.9218121f, rf * fmaf(rf, B, A));
  return fma(r, c2, C1);
}
// 2^(floor(k/1024) + (k mod 1024)/1024) for exponents in the normal range
__device__ __forceinline__ double exp2_int(int k) {
  return scale2(__ldg(&kExp2Tab[k & 1023].t), k >> 10);
}
// a 2^((k + r)/1024), the table's rounding error taken out: a t (1 + (r u + d))
__device__ __forceinline__ double exp2_times(double a, int k, double r) {
  const double2 e = __ldg(reinterpret_cast<const double2 *>(&kExp2Tab[k & 1023]));
  const double t = a * scale2(e.x, k >> 10);
  return fma(t, fma(r, exp2_slope(r), e.y), t);
}
// 2^((k + r)/1024); exponents below -1000 give zero (every caller's result is then below 1e-99)
__device__ __forceinline__ double exp2k(int k, double r) {
  const double2 e = __ldg(reinterpret_cast<const double2 *>(&kExp2Tab[k & 1023]));
  const double t = scale2(e.x, k >> 10);
  return k < -1000 * 1024 ? 0.0 : fma(t, fma(r, exp2_slope(r), e.y), t);
}
// exp(x) for |x| < 700, to zero below
__device__ __forceinline__ double exp_fast(double x) {
  const float xf = d2f(x);
  float kf;
  const int k = rint_f(fmaxf(xf, -700.0f) * (float)K_LN2, kf);
  double r = fma(x, K_LN2, flip(f2d(kf)));
  r = fma(x, (double)K_LN2_LO, r);
  return xf < -700.0f ? 0.0 : exp2k(k, r);
}

// 1024 log2(x) = h + l for positive normal x (l < 1e-2)
struct Log2 {
  double h, l;
};
__device__ __forceinline__ Log2 log2k(double x) {
  const int hx = hi32(x);
  const int e = (hx >> 20) - 1023;
  const LogRow *row = &kLogTab[(hx >> 11) & 511];
  const double th = __ldg(&row->hi);
  const float2 cl = __ldg(reinterpret_cast<const float2 *>(&row->c));
  const double m = __hiloint2double((hx & 0xfffff) | 0x3ff00000, lo32(x));
  const double r = fma(m, f2d(cl.x), -1.0);       // exact but for 2^-63
  const double a = f2d((float)(e * 1024)) + th;   // exact
  const double b = r * K_LN2;
  const float rf = d2f(r);
  const float bl = fmaf(rf, K_LN2_LO, cl.y);
  const double be = fma(r, K_LN2, -b);
  Log2 L;
  L.h = a + b;                                     // |a| > |b|, or a = 0
  const double t = (b - (L.h - a)) + be;
  // -r^2/2 + r^3/3 - r^4/4 + r^5/5, times 1024/ln 2: the cubic coefficient carries the rest
  const double c3 = add_rel(K_LN2 / 3.0, 1.9235934f, rf * fmaf(rf, 0.6f, -0.75f));
  L.l = fma(r * r, fma(r, c3, -0.5 * K_LN2), t) + f2d(bl);
  return L;
}
// log10(x) to one double (0.545 ulp for x of 1e12 and more), x positive normal: the
// row's exact part times log10(2)/1024 and the series, already in tens, in the
// last sum alone
__device__ __forceinline__ double log10_fast(double x) {
  constexpr double LG = 0.00029397460514060664;   // log10(2)/1024, to 9e-18 of it
  constexpr double M = 0.43429448190325182;       // 1/ln 10
  const int hx = hi32(x);
  const int e = (hx >> 20) - 1023;
  const LogRow *row = &kLogTab[(hx >> 11) & 511];
  const double m = __hiloint2double((hx & 0xfffff) | 0x3ff00000, lo32(x));
  const float2 cl = __ldg(reinterpret_cast<const float2 *>(&row->c));
  const double r = fma(m, f2d(cl.x), -1.0);
  const double a = f2d((float)(e * 1024)) + __ldg(&row->hi);   // exact
  const float rf = d2f(r);
  // (1/ln 10) (1 - r/2 + r^2/3 - r^3/4)
  const double c2 = add_rel(-0.5 * M, 1.7371779f, rf * fmaf(rf, fmaf(rf, -0.4f, 0.5f), -2.0f / 3.0f));
  return fma(a, LG, fma(r, fma(r, c2, M), f2d(cl.y * (float)LG)));
}
// b L -> the integer k and remainder r of 1024 log2(x^b); returns k
__device__ __forceinline__ int pow_arg(const Log2 &L, double b, double &r) {
  float kf;
  const int k = rint_f(d2f(b) * d2f(L.h), kf);
  r = fma(b, L.l, fma(b, L.h, flip(f2d(kf))));
  return k;
}
// x^b from L = log2k(x), |b log2 x| < 1000
__device__ __forceinline__ double powk(const Log2 &L, double b) {
  double r;
  const int k = pow_arg(L, b, r);
  return exp2k(k, r);
}

// 1/b to about 2^-44 from the FP32 unit, without an FP64 operation; b normal, its result too
__device__ __forceinline__ double rcp_seed(double b) {
  const unsigned h = (unsigned)hi32(b), l = (unsigned)lo32(b);
  // the mantissa as bh + bl, 24 + 24 bits
  const float bh = __uint_as_float((__funnelshift_l(l, h, 3) & 0x7fffffu) | 0x3f800000u);
  const float bl = (float)((l & 0x1fffffffu) >> 5) * 7.105427357601002e-15f;   // 2^-47
  float y0 = rcp_approx(bh);
  y0 = fminf(fmaxf(y0, 0.5f), 0.99999994f);        // 1/b is in (1/2, 1]
  const float e = fmaf(-bl, y0, fmaf(-bh, y0, 1.0f));
  const float y1 = fmaf(y0 * e, e, y0 * e);
  // y0 + y1 in y0's mantissa (y1 is below 2^-20 of it), the exponent and sign of b taken out
  const unsigned u = __float_as_uint(y0);
  const long long be = (long long)((h >> 20) & 0x7ff) - 1023;
  long long bits = ((long long)(u >> 3) << 32 | (long long)(unsigned)(u << 29)) + 0x3800000000000000ll - (be << 52);
  bits += (long long)__float2int_rn(y1 * 2251799813685248.0f) << 2;             // 2^51
  return __longlong_as_double(bits | (long long)((unsigned long long)(h & 0x80000000u) << 32));
}
// 1/b within 0.5 + 2^-35 ulp (2 FP64 instructions where the operand and result
// are normal; the terms left out are 2^-88 of the result, so one in about 2^35
// rounds the other way.  Settled like the square root below it cost 20,011 CO
// cells 5 %, 3.10 -> 3.25 ms, and 1,500 cells of FP64 chemistry 2 %.)
__device__ __forceinline__ double rcp_near(double b) {
  const unsigned e = ((unsigned)hi32(b) >> 20) & 0x7ff;
  if (e - 2u >= 2042u) return __drcp_rn(b);   // zero, denormal, infinite, NaN, or a denormal result
  const double y = rcp_seed(b);
  return fma(y, fma(-b, y, 1.0), y);
}
// a/b for normal operands and result: within 0.5 + 2^-35 ulp, as rcp_near
__device__ __forceinline__ double div_fast(double a, double b) {
  const double y = rcp_seed(b);
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}
// a/b: div_fast where both and the quotient are normal with room, else the division
__device__ __forceinline__ double div_any(double a, double b) {
  const unsigned ea = ((unsigned)hi32(a) >> 20) & 0x7ff, eb = ((unsigned)hi32(b) >> 20) & 0x7ff;
  if (ea - 64u > 1918u || eb - 64u > 1918u || ea - eb + 959u > 1918u) return a / b;
  return div_fast(a, b);
}
// q, within 1.4 ulp of the exact result, or the neighbour that is nearer to it: res is the exact residual of q, whose magnitude passes `half`
// (the bits of a positive value) where the exact result lies half an ulp beyond
// q.  Below a power of two the ulp is half as large.  Integer operations only.
__device__ __forceinline__ double settle(double q, double res, long long half) {
  const long long r = __double_as_longlong(res), mag = r & 0x7fffffffffffffffll, qb = __double_as_longlong(q);
  const long long below = half - ((qb & 0xfffffffffffffll) ? 0ll : 1ll << 52);
  return __longlong_as_double(qb + (r >= 0 ? (mag > half ? 1 : 0) : (mag >= below ? -1 : 0)));
}
// sqrt(x), rounded: five FP64 instructions where x is within FP32's normal range.
// From y near 1/sqrt(x), g = x y and r = (1 - x y^2)/2 < 2^-20, the root is
// g (1 + r + 3 r^2/2 + ...), to 2^-62 and the rounding of g; the exact residual
// x - g^2 settles it: at the midpoint above g it is g ulp(g) + ulp(g)^2/4, in whole
// ulp(g)^2 beyond it.
__device__ __forceinline__ double sqrt_rn(double x) {
  if ((unsigned)hi32(x) - 0x38200000u > 0x0f000000u) return __dsqrt_rn(x);   // zero, negative, tiny, huge, NaN
  const float y0 = rsqrt_approx(d2f(x));
  const double y = f2d(y0), g = x * y;
  const double r = fma(-g, scale2(y, -1), 0.5);
  const double g1 = fma(g, fma(r, f2d(1.5f * d2f(r)), r), g);
  const long long eg = (long long)((unsigned)hi32(g1) >> 20) - 1023;
  return settle(g1, fma(-g1, g1, x), __double_as_longlong(g1) + (eg - 52) * (1ll << 52));
}
// 1/sqrt(x), x positive normal within FP32's range
__device__ __forceinline__ double rsqrt_fast(double x) {
  const float y0 = rsqrt_approx(d2f(x));
  const double y = f2d(y0 * 0.9999996f);            // from below, so that e > 0
  const double e = fma(-(x * y), y, 1.0);
  // y (1 + e/2 + 3 e^2/8), e < 2^-18
  return fma(y * e, add_rel(0.5, 1.0f, 0.75f * d2f(e)), y);
}

}  // namespace fp64
}  // namespace pdr
