// Double-float (pairs of floats) arithmetic: complex operations, division,
// sine, cosine and sinc, the CTA-wide FFT and reduction, and the
// result write of the double-float re-evaluation of mixed proposals
// (ucb_fd_hp.cu).
#pragma once
#include "glass_common.cuh"

namespace glass {

struct dc {
  df re, im;
};
__device__ __forceinline__ dc dc_add(dc a, dc b) { return {df_add(a.re, b.re), df_add(a.im, b.im)}; }
__device__ __forceinline__ dc dc_sub(dc a, dc b) { return {df_add(a.re, df_neg(b.re)), df_add(a.im, df_neg(b.im))}; }
// a b + c d: the two exact products summed before the one renormalisation
__device__ __forceinline__ df df_mul2_add(df a, df b, df c, df d) {
  const df p = two_prod(a.hi, b.hi), q = two_prod(c.hi, d.hi), s = two_sum(p.hi, q.hi);
  const float l = __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, p.lo));
  const float m = __fmaf_rn(c.hi, d.lo, __fmaf_rn(c.lo, d.hi, q.lo));
  return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(l, m)));
}
__device__ __forceinline__ dc dc_mul(dc a, dc b) {
  return {df_mul2_add(a.re, b.re, df_neg(a.im), b.im), df_mul2_add(a.re, b.im, a.im, b.re)};
}
__device__ __forceinline__ dc dc_mi(dc a) { return {a.im, df_neg(a.re)}; }  // -i a
// complex hi + lo floats (x, y: hi; z, w: lo), as the tables store them: no
// FP64 conversion in the inner loops (GB300's FP64 pipe runs at 1/64 rate)
__device__ __forceinline__ dc dc_from(float4 v) { return {{v.x, v.z}, {v.y, v.w}}; }
__device__ __forceinline__ dc dc_from(float2 hi, float2 lo) { return {{hi.x, lo.x}, {hi.y, lo.y}}; }
__device__ __forceinline__ df df_sq_sum(dc a) { return df_mul2_add(a.re, a.re, a.im, a.im); }
// a times an exact power of two
__device__ __forceinline__ dc dc_scale2(dc a, float p2) {
  return {{a.re.hi * p2, a.re.lo * p2}, {a.im.hi * p2, a.im.lo * p2}};
}

// Double-float division (one Newton correction of the float quotient).
__device__ __forceinline__ df df_div(df a, df b) {
  const float q1 = __fdiv_rn(a.hi, b.hi);
  const df r = df_add(a, df_neg(df_mul_f(b, q1)));
  return quick_two_sum(q1, __fdiv_rn(r.hi, b.hi));
}

// Inverse factorials 1/n! as hi + lo floats, n = 0..19 (the Taylor
// coefficients of sin and cos).
__device__ __forceinline__ df inv_fact(int n) {
  switch (n) {
    case 0: case 1: return {1.f, 0.f};
    case 2: return {0.5f, 0.f};
    case 3: return {0.1666666716337204f, -4.967053879312289e-09f};
    case 4: return {0.0416666679084301f, -1.2417634698280722e-09f};
    case 5: return {0.008333333767950535f, -4.34617203337595e-10f};
    case 6: return {0.0013888889225199819f, -3.3631094437103215e-11f};
    case 7: return {0.00019841270113829523f, -2.725596874933456e-12f};
    case 8: return {2.4801587642286904e-05f, -3.40699609366682e-13f};
    case 9: return {2.7557318844628753e-06f, 3.793571224297229e-14f};
    case 10: return {2.755731998149713e-07f, -7.575112209051195e-15f};
    case 11: return {2.5052107943679403e-08f, 4.4176230446483665e-16f};
    case 12: return {2.0876755879584152e-09f, 1.1082839147459852e-16f};
    case 13: return {1.6059044372074283e-10f, -5.352526511562726e-18f};
    case 14: return {1.147074536050896e-11f, 2.372207689231238e-19f};
    case 15: return {7.647163609812713e-13f, 1.2200710471178288e-20f};
    case 16: return {4.7794772561329454e-14f, 7.62544404448643e-22f};
    case 17: return {2.8114573589663704e-15f, -1.0462084739763658e-22f};
    case 18: return {1.5619206814541513e-16f, 1.5404471465941993e-24f};
    default: return {8.220635078476521e-18f, 1.681478096855898e-25f};
  }
}

// sum_k (-1)^k x2^k / (2k + first)!, k = 0..terms-1, by Horner in
// double-float (first = 1: sin(x)/x; first = 0: cos x).
template <int FIRST, int TERMS>
__device__ __forceinline__ df df_alt_series(df x2) {
  df p = inv_fact(2 * (TERMS - 1) + FIRST);
  if ((TERMS - 1) & 1) p = df_neg(p);
#pragma unroll
  for (int k = TERMS - 2; k >= 0; k--) {
    df c = inv_fact(2 * k + FIRST);
    if (k & 1) c = df_neg(c);
    p = df_add(df_mul(p, x2), c);
  }
  return p;
}

// sin and cos of a double-float angle with a table: tab[k] = (sin, cos) of
// k pi/32 as hi + lo floats (float4: sin hi, sin lo, cos hi, cos lo), k mod
// 64; x = k pi/32 + d with |d| <= pi/64 (three-part pi/32), whose sine
// (through d^7) and cosine (through d^8) have truncation errors below 1e-15;
// then the angle-sum formulas.
__device__ __forceinline__ void df_sincos_tab(df x, const float4 *tab, df *s, df *c) {
  const float q = rintf(x.hi * 10.185916357881302f);  // 32/pi
  df d = df_add(x, df_neg(two_prod(q, 0.09817477315664291f)));
  d = df_add(d, df_neg(two_prod(q, -2.7319617679211206e-09f)));
  d = df_add(d, df{q * 1.0719528187536762e-16f, 0.f});
  const df d2 = df_mul(d, d);
  const df sd = df_mul(d, df_alt_series<1, 4>(d2));
  const df cd = df_alt_series<0, 5>(d2);
  const float4 t = tab[((int)q) & 63];
  const df sk = {t.x, t.y}, ck = {t.z, t.w};
  *s = df_add(df_mul(sk, cd), df_mul(ck, sd));
  *c = df_add(df_mul(ck, cd), df_neg(df_mul(sk, sd)));
}

// sin(x)/x in double-float: Taylor series through x^12 for |x| <= 1/2 and
// through x^18 for |x| <= 1 (truncation below 1e-17), sin x / x beyond.
__device__ __forceinline__ df df_sinc(df x, const float4 *tab) {
  const float ax = fabsf(x.hi);
  if (ax <= 0.5f) return df_alt_series<1, 7>(df_mul(x, x));
  if (ax <= 1.f) return df_alt_series<1, 10>(df_mul(x, x));
  df s, c;
  df_sincos_tab(x, tab, &s, &c);
  return df_div(s, x);
}

// In-place FFT of nser series of N = 2^ln double-floats, back to back, by the CTA:
// decimation in time from digit-reversed order (element n of series s at hp_at(s N +
// hp_rev(n, ln))), radix-4 stages (sub-transform size p: butterfly i < nser N/4, k =
// i mod p, on x[4 (i - k) + k + m p] times exp(-2 pi i m k / (4p)), m = 0..3) and a
// final radix-2 stage when log2 N is odd; results in natural order at hp_at.  tw[j] =
// exp(-2 pi i j / N) as hi + lo floats, read from global memory (L1 after the first
// touch): 16 bytes of shared memory per point.
//
// hp_at: a 16-byte access serves 8 lanes at a time, one per 16-byte column; the
// permutation within each run of 8 elements puts the strides of the first stages
// (4 and 16) and of the digit-reversed scatter on different columns.
__device__ __forceinline__ int hp_at(int i) {
  return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9) ^ ((i >> 2) & 4)) & 7);
}
// base-4 digits of n reversed; with ln odd the lowest bit becomes the highest
// (the radix-2 stage's digit)
__device__ __forceinline__ int hp_rev(int n, int ln) {
  const int top = (ln & 1) ? (n & 1) << (ln - 1) : 0;
  const int l4 = ln & ~1, m = (ln & 1) ? n >> 1 : n;
  const unsigned r = __brev((unsigned)m) >> (32 - l4);
  return top + (int)(((r & 0x55555555u) << 1) | ((r >> 1) & 0x55555555u));
}
// A radix-4 butterfly (w1, w2, w3: its factors, where it has any).
__device__ __forceinline__ void hp_radix4(dc *x0, dc *x1, dc *x2, dc *x3, dc u0, dc u1, dc u2, dc u3, bool factors,
                                          float4 w1, float4 w2, float4 w3) {
  if (factors) {
    u1 = dc_mul(u1, dc_from(w1));
    u2 = dc_mul(u2, dc_from(w2));
    u3 = dc_mul(u3, dc_from(w3));
  }
  const dc a = dc_add(u0, u2), b = dc_sub(u0, u2), c = dc_add(u1, u3), d = dc_mi(dc_sub(u1, u3));
  *x0 = dc_add(a, c);
  *x1 = dc_add(b, d);
  *x2 = dc_sub(a, c);
  *x3 = dc_sub(b, d);
}
// The twiddles of a thread's next butterfly (of its next stage, after the last of
// one) are loaded before the arithmetic of the current one: each is used once per
// series, so every load is a trip to L2.  One copy for clusters and single CTAs: with
// a copy each, fetching the kernel's instructions cost a step that starts with cold
// caches 0.9 us.
static __device__ __noinline__ void hp_fft(dc *x, int ln, int nser, const float4 *__restrict__ tw) {
  const int N = 1 << ln, Q = nser * N / 4;  // Q radix-4 butterflies a stage
  float4 w[3] = {};
  int lp = 0;
  for (; lp + 2 <= ln; lp += 2) {
    const int p = 1 << lp;
    for (int i = threadIdx.x; i < Q; i += blockDim.x) {
      const int k = i & (p - 1), j = ((i - k) << 2) + k;
      dc *const x0 = x + hp_at(j), *const x1 = x + hp_at(j + p), *const x2 = x + hp_at(j + 2 * p),
               *const x3 = x + hp_at(j + 3 * p);
      const dc u0 = *x0, u1 = *x1, u2 = *x2, u3 = *x3;
      const float4 w1 = w[0], w2 = w[1], w3 = w[2];
      const bool last = i + (int)blockDim.x >= Q;
      const int lq = last ? lp + 2 : lp, in = last ? (int)threadIdx.x : i + (int)blockDim.x;
      if (lq + 2 <= ln) {
        const int kn = (in & ((1 << lq) - 1)) << (ln - lq - 2);
        if (lq > 0) {
          w[0] = tw[kn];
          w[1] = tw[2 * kn];
          w[2] = tw[3 * kn];
        }
      } else if (lq < ln) {
        w[0] = tw[in & (N / 2 - 1)];  // the radix-2 stage's first
      }
      hp_radix4(x0, x1, x2, x3, u0, u1, u2, u3, lp > 0, w1, w2, w3);
    }
    __syncthreads();
  }
  if (lp < ln) {  // log2 N odd: one radix-2 stage, p = N/2
    if ((int)threadIdx.x >= Q && (int)threadIdx.x < 2 * Q) w[0] = tw[threadIdx.x & (N / 2 - 1)];
    for (int i = threadIdx.x; i < 2 * Q; i += blockDim.x) {
      const int k = i & (N / 2 - 1), j = ((i - k) << 1) + k;
      dc *const x0 = x + hp_at(j), *const x1 = x + hp_at(j + N / 2);
      const float4 w1 = w[0];
      if (i + (int)blockDim.x < 2 * Q) w[0] = tw[(i + blockDim.x) & (N / 2 - 1)];
      const dc a = *x0, b = dc_mul(*x1, dc_from(w1));
      *x0 = dc_add(a, b);
      *x1 = dc_sub(a, b);
    }
    __syncthreads();
  }
}

// Sum over the CTA of a double-float per thread (valid in thread 0).
static __device__ df hp_block_sum(df v, float2 *red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    df o = {__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off)};
    v = df_add(v, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(v.hi, v.lo);
  __syncthreads();
  df t = {0.f, 0.f};
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t = df_add(t, df{red[w].x, red[w].y});
  return t;
}

// Writes a re-evaluated proposal's results (thread 0), as the spectral
// kernels do; returns term_y.
__device__ __forceinline__ double hp_write(int item, int N, int seg, int imin, int NFFT, const df s[3],
                                           const double *Q, const double *QA, bool perch, const double *term_x,
                                           double *dlogl, double *term_y, double *hh, double *term_ch,
                                           int *status) {
  const int jlo = imin < 0 ? 0 : imin;
  const int jhi = imin + N > NFFT ? NFFT : imin + N;
  const double *Qs = Q + (size_t)seg * (NFFT + 1);
  double term;
  if (perch) {
    const double *QAs = QA + (size_t)seg * (NFFT + 1);
    const double qa = QAs[jhi] - QAs[jlo];
    const double tA = (qa - (double)s[0].hi) - (double)s[0].lo;
    const double tE = (((Qs[jhi] - Qs[jlo]) - qa) - (double)s[1].hi) - (double)s[1].lo;
    term_ch[2 * (size_t)item] = tA;
    term_ch[2 * (size_t)item + 1] = tE;
    term = tA + tE;
  } else {
    const df r = df_add(s[0], s[1]);
    term = ((Qs[jhi] - Qs[jlo]) - (double)r.hi) - (double)r.lo;
  }
  const double tx = term_x ? term_x[item] : 0.0;
  dlogl[item] = term - tx;
  if (term_y) term_y[item] = term;
  if (hh) hh[item] = 2.0 * ((double)s[2].hi + (double)s[2].lo);
  if (status) status[item] = isfinite(term) ? 0 : 1;
  return term;
}

}  // namespace glass
