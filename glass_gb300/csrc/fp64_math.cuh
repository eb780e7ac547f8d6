// FP64 building blocks counted in FP64 instructions.
//
// GB300's FP64 pipe does 2 multiply-adds per SM and clock, 1/64 of FP32: a
// warp's FP64 instruction holds it for 16 clocks, and integer work, loads and
// selects are free beside it.  The forms here spend table loads and integer
// operations to save FP64 instructions, at the accuracy of the library's.
#pragma once
#include <math.h>

namespace glass {

// 1/x for normal x of moderate exponent: the hardware's ~20-bit estimate and
// one step of Householder's cubic iteration, r (1 + e + e^2) with e = 1 - x r.
__device__ __forceinline__ double rcp_fast(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// a / b from rb = 1/b: the product and one exact-residual step (3 FP64 instructions
// instead of about 9).  Before its rounding the result is within 2^-104 of the
// quotient, relatively (2^-102 where rb is good to a few ulp only): the last bit can
// differ from the quotient's where that lies so close to the middle of two doubles.
__device__ __forceinline__ double div_by(double a, double b, double rb) {
  const double q = a * rb;
  return fma(fma(-q, b, a), rb, q);
}

constexpr double kRoundMagic = 6755399441055744.0;  // 1.5 2^52: adding it rounds to the nearest integer

// exp by table and short polynomial (Tang, ACM Trans. Math. Softw. 15, 1989):
// x = (64 m + k) ln2/64 + r, exp x = 2^m t[k] (1 + r + ... + r^5/120), t[k] =
// 2^(k/64), |r| <= ln2/128.  10 FP64 instructions; arguments beyond +-708 and
// NaN go to the library's.
constexpr int kExpTab = 64;
__device__ __forceinline__ double exp_tab(double x, const double *t) {
  if ((__double2hiint(x) & 0x7fffffff) >= 0x40862000) return exp(x);
  constexpr double kLn2 = 0.693147180559945309417, kLn2Lo = 2.3190468138462996e-17;  // ln 2 = kLn2 + kLn2Lo
  const double z = fma(x, kExpTab / kLn2, kRoundMagic);
  const int n = __double2loint(z);
  const double kd = z - kRoundMagic;
  double r = fma(kd, -kLn2 / kExpTab, x);
  r = fma(kd, -kLn2Lo / kExpTab, r);
  double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  q = fma(r, q, 1.0 / 6.0);
  q = fma(r, q, 0.5);
  q = fma(r * r, q, r);
  const double T = t[n & (kExpTab - 1)];
  const double y = fma(T, q, T);
  return __hiloint2double(__double2hiint(y) + ((n >> 6) << 20), __double2loint(y));
}
__device__ __forceinline__ void exp_tab_fill(double *t) {
  for (int k = threadIdx.x; k < kExpTab; k += blockDim.x) t[k] = exp2(k * (1.0 / kExpTab));
}

// sin x and cos x by table and short polynomials (the same method): x = k
// 2 pi/1024 + r, |r| <= pi/1024, and the angle-sum formulas.  tw: the 1024-point
// FFT twiddles exp(-2 pi i k/1024).  14 FP64 instructions (the library's take
// about 25, and more beyond 1e5); within 1 ulp of 1 like theirs.  x - k (2 pi/1024),
// with the constant's first 53 bits, is exact, and the next 53 leave 1e-17 up to
// |x| = 1e7; larger and non-finite x go to the library's.
constexpr int kSincosTab = 1024;
__device__ __forceinline__ void sincos_tab(double x, const double2 *tw, double *s, double *c) {
  if ((__double2hiint(x) & 0x7fffffff) >= 0x416312d0) {
    sincos(x, s, c);
    return;
  }
  constexpr double k2Pi = 6.283185307179586477, k2PiLo = 2.4492935982947064e-16;  // 2 pi = k2Pi + k2PiLo
  const double z = fma(x, kSincosTab / k2Pi, kRoundMagic);
  const double kd = z - kRoundMagic;
  double r = fma(kd, -k2Pi / kSincosTab, x);
  r = fma(kd, -k2PiLo / kSincosTab, r);
  const double2 t = tw[__double2loint(z) & (kSincosTab - 1)];  // cos, -sin of the table angle
  const double r2 = r * r;
  const double sn = fma(r * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), r);
  const double cm1 = r2 * fma(r2, 1.0 / 24.0, -0.5);
  *c = fma(t.y, sn, fma(t.x, cm1, t.x));
  *s = fma(t.x, sn, -fma(t.y, cm1, t.y));
}

// cos x alone: 12 FP64 instructions.
__device__ __forceinline__ double cos_tab(double x, const double2 *tw) {
  if ((__double2hiint(x) & 0x7fffffff) >= 0x416312d0) return cos(x);
  constexpr double k2Pi = 6.283185307179586477, k2PiLo = 2.4492935982947064e-16;
  const double z = fma(x, kSincosTab / k2Pi, kRoundMagic);
  const double kd = z - kRoundMagic;
  double r = fma(kd, -k2Pi / kSincosTab, x);
  r = fma(kd, -k2PiLo / kSincosTab, r);
  const double2 t = tw[__double2loint(z) & (kSincosTab - 1)];
  const double r2 = r * r;
  const double sn = fma(r * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), r);
  return fma(t.y, sn, fma(t.x, r2 * fma(r2, 1.0 / 24.0, -0.5), t.x));
}

// sin(x) / x: the Taylor series for |x| <= 1 (to x^10/11! for |x| <= 0.2, to
// x^16/17! beyond: truncation below 1e-17), else the quotient.
__device__ __forceinline__ double sinc64(double x) {
  const double z = x * x;
  const int h = __double2hiint(z);
  if (h <= 0x3fa47ae1) {  // z <= 0.04
    double p = fma(z, -1.0 / 39916800.0, 1.0 / 362880.0);
    p = fma(z, p, -1.0 / 5040.0);
    p = fma(z, p, 1.0 / 120.0);
    p = fma(z, p, -1.0 / 6.0);
    return fma(z, p, 1.0);
  }
  if (h < 0x3ff00000) {  // z < 1
    double p = fma(z, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);
    p = fma(z, p, 1.0 / 6227020800.0);
    p = fma(z, p, -1.0 / 39916800.0);
    p = fma(z, p, 1.0 / 362880.0);
    p = fma(z, p, -1.0 / 5040.0);
    p = fma(z, p, 1.0 / 120.0);
    p = fma(z, p, -1.0 / 6.0);
    return fma(z, p, 1.0);
  }
  return sin(x) / x;
}

// x truncated to an integer (through 64 bits), as a double.
__device__ __forceinline__ double trunc_i64(double x) { return (double)(long long)x; }

// x 2^e of a normal x with a normal result by exponent arithmetic, else scalbn.
__device__ __forceinline__ double scale_pow2(double x, int e) {
  const int k = (__double2hiint(x) >> 20) & 0x7ff;
  if (k == 0 || k == 0x7ff || k + e <= 0 || k + e >= 0x7ff) return scalbn(x, e);
  return __hiloint2double(__double2hiint(x) + (e << 20), __double2loint(x));
}

// The float nearest x (ties to even) by integer arithmetic, for 2^-123 <= |x| <
// 2^127 (conversions between FP64 and FP32 run at the FP64 pipe's rate); the
// double of such a float.
__device__ __forceinline__ float f32_nearest(double x) {
  const unsigned long long b = __double_as_longlong(x), a = b & 0x7fffffffffffffffull;
  const unsigned f = (unsigned)(((a + 0x0fffffffull + ((a >> 29) & 1)) >> 29) - (896ull << 23));
  return __uint_as_float(f | ((unsigned)(b >> 32) & 0x80000000u));
}
__device__ __forceinline__ double f64_of(float x) {
  const unsigned f = __float_as_uint(x);
  const unsigned long long a = ((unsigned long long)(f & 0x7fffffffu) + (896ull << 23)) << 29;
  return __longlong_as_double(a | ((unsigned long long)(f & 0x80000000u) << 32));
}
// hi + lo floats of x, as (float)x and (float)(x - (double)hi), with one FP64
// instruction; the conversions for |x| outside [2^-68, 2^127).
__device__ __forceinline__ void split_f32(double x, float &hi, float &lo) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ff;
  if (e - 955u >= 194u) {  // beyond [2^-68, 2^126), where every step below is normal or zero
    hi = (float)x;
    lo = (float)(x - (double)hi);
    return;
  }
  hi = f32_nearest(x);
  const double r = x - f64_of(hi);  // exact: 0, or at least 2^-53 |x|
  lo = __double_as_longlong(r) << 1 ? f32_nearest(r) : 0.f;
}
// (float)x alone.
__device__ __forceinline__ float to_f32(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ff;
  return e - 903u >= 246u ? (float)x : f32_nearest(x);
}

// FFT factors in tangent form (Linzer and Feig, IEEE Trans. Signal Process. 41,
// 1993): c + i y is kept as (c, t = y / c), so that a +- (c + i y) b = a +- c (b.x - t
// b.y + i (b.y + t b.x)) takes 6 multiply-adds, where the product and the sums
// take 8, and a radix-4 butterfly, as two levels of these with the factors w
// and w^2, 24 where it takes 28 with w, w^2 and w^3.  The rounding of t is a
// relative one of y, so no angle loses accuracy; at c = 0, c = 2^-60 stands in.
__host__ __device__ inline double2 tan_form(double c, double y) {
  if (fabs(c) < 1e-15) c = 1.0 / 1152921504606846976.0;
  return make_double2(c, y / c);
}
__device__ __forceinline__ double2 tan_mul(double2 b, double2 w) {
  return make_double2(w.x * fma(-w.y, b.y, b.x), w.x * fma(w.y, b.x, b.y));
}
// p, m = a +- w b
__device__ __forceinline__ void tan_radix2(double2 a, double2 b, double2 w, double2 &p, double2 &m) {
  const double u = fma(-w.y, b.y, b.x), v = fma(w.y, b.x, b.y);
  p = make_double2(fma(w.x, u, a.x), fma(w.x, v, a.y));
  m = make_double2(fma(-w.x, u, a.x), fma(-w.x, v, a.y));
}
// The 4-point DFT (sign -1: forward) of v0, w v1, w^2 v2, w^3 v3; w2 = w^2.
template <int SIGN>
__device__ __forceinline__ void tan_radix4(double2 &v0, double2 &v1, double2 &v2, double2 &v3, double2 w, double2 w2) {
  double2 a, b, p, q;
  tan_radix2(v0, v2, w2, a, b);
  tan_radix2(v1, v3, w2, p, q);
  tan_radix2(a, p, w, v0, v2);
  const double u = w.x * SIGN, r = fma(-w.y, q.y, q.x), i = fma(w.y, q.x, q.y);  // b +- SIGN i w q
  v1 = make_double2(fma(-u, i, b.x), fma(u, r, b.y));
  v3 = make_double2(fma(u, i, b.x), fma(-u, r, b.y));
}
// The same with w = 1: 16 additions.
template <int SIGN>
__device__ __forceinline__ void plain_radix4(double2 &v0, double2 &v1, double2 &v2, double2 &v3) {
  const double2 a = make_double2(v0.x + v2.x, v0.y + v2.y), b = make_double2(v0.x - v2.x, v0.y - v2.y);
  const double2 p = make_double2(v1.x + v3.x, v1.y + v3.y), q = make_double2(v1.x - v3.x, v1.y - v3.y);
  v0 = make_double2(a.x + p.x, a.y + p.y);
  v2 = make_double2(a.x - p.x, a.y - p.y);
  v1 = SIGN < 0 ? make_double2(b.x + q.y, b.y - q.x) : make_double2(b.x - q.y, b.y + q.x);
  v3 = SIGN < 0 ? make_double2(b.x - q.y, b.y + q.x) : make_double2(b.x + q.y, b.y - q.x);
}

}  // namespace glass
