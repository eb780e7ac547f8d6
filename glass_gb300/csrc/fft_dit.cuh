// In-place mixed-radix FFTs in shared memory, the whole CTA on each.
#pragma once
#include <cuda_runtime.h>

#include "fp64_math.cuh"

namespace glass {
namespace {

// Radices of an in-place decimation-in-time FFT: 3s, then 4s, then a 2.
struct RadixPlan {
  int n;
  int r[24];
  int pre[24];  // R_0 ... R_{s-1}
};

__device__ __forceinline__ void radix_plan(int L, RadixPlan &P) {
  P.n = 0;
  int rem = L, pre = 1;
  while (rem % 3 == 0) {
    P.r[P.n] = 3;
    P.pre[P.n++] = pre;
    pre *= 3;
    rem /= 3;
  }
  while (rem % 4 == 0) {
    P.r[P.n] = 4;
    P.pre[P.n++] = pre;
    pre *= 4;
    rem /= 4;
  }
  while (rem % 2 == 0) {
    P.r[P.n] = 2;
    P.pre[P.n++] = pre;
    pre *= 2;
    rem /= 2;
  }
}

// Input position of element x: its stage digits read in reverse.
__device__ __forceinline__ int digit_rev(int x, const RadixPlan &P) {
  int pos = 0;
  for (int s = P.n - 1; s >= 0; s--) {
    const int d = x % P.r[s];
    x /= P.r[s];
    pos += d * P.pre[s];
  }
  return pos;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C>
__device__ __forceinline__ C mkc(decltype(C::x) x, decltype(C::x) y) {
  C r;
  r.x = x;
  r.y = y;
  return r;
}

// In-place mixed-radix FFTs of nser series a[L], back to back, each held in
// digit-reversed order; results in natural order.  tw[j * twmul] = e^{-2 pi i j /
// L}, in FP64 in tangent form (tan_form); SIGN -1 forward, +1 inverse
// (unnormalised).  Whole CTA.  C = double2 or float2.  In FP64 3 instructions
// per point and factor of two (24 per radix-4 butterfly), the first stage without
// its factors.
template <int SIGN, typename C>
__device__ void dit_fft(C *a, int L, const RadixPlan &P, const C *__restrict__ tw, int twmul, int nser = 1) {
  constexpr int sign = SIGN;
  using R = decltype(C::x);
  constexpr bool kF64 = sizeof(R) == 8;
  int p = 1;
  for (int st = 0; st < P.n; st++) {
    const int Rd = P.r[st], q = p * Rd, nb = L / Rd;
    const int tstep = (L / q) * twmul;
    for (int t = threadIdx.x; t < nb * nser; t += blockDim.x) {  // series of L = nb Rd points: b counts on
      const int b = t / p, k = t - b * p;
      const int i0 = b * q + k;
      C *const x0 = a + i0, *const x1 = a + i0 + p;
      if (Rd == 4) {
        C *const x2 = a + i0 + 2 * p, *const x3 = a + i0 + 3 * p;
        C v0 = *x0, v1 = *x1, v2 = *x2, v3 = *x3;
        if constexpr (kF64) {
          if (st > 0) {
            C w1 = tw[k * tstep], w2 = tw[2 * k * tstep];
            if (sign > 0) {
              w1.y = -w1.y;
              w2.y = -w2.y;
            }
            tan_radix4<SIGN>(v0, v1, v2, v3, w1, w2);
          } else {  // the first stage's factors are 1
            plain_radix4<SIGN>(v0, v1, v2, v3);
          }
          *x0 = v0;
          *x1 = v1;
          *x2 = v2;
          *x3 = v3;
        } else {
          C w1 = tw[k * tstep], w2 = tw[2 * k * tstep], w3 = tw[3 * k * tstep];
          if (sign > 0) {
            w1.y = -w1.y;
            w2.y = -w2.y;
            w3.y = -w3.y;
          }
          v1 = cmul(v1, w1);
          v2 = cmul(v2, w2);
          v3 = cmul(v3, w3);
          const C t0 = mkc<C>(v0.x + v2.x, v0.y + v2.y), t1 = mkc<C>(v0.x - v2.x, v0.y - v2.y);
          const C t2 = mkc<C>(v1.x + v3.x, v1.y + v3.y), t3 = mkc<C>(v1.x - v3.x, v1.y - v3.y);
          const C t3r = sign < 0 ? mkc<C>(t3.y, -t3.x) : mkc<C>(-t3.y, t3.x);
          *x0 = mkc<C>(t0.x + t2.x, t0.y + t2.y);
          *x1 = mkc<C>(t1.x + t3r.x, t1.y + t3r.y);
          *x2 = mkc<C>(t0.x - t2.x, t0.y - t2.y);
          *x3 = mkc<C>(t1.x - t3r.x, t1.y - t3r.y);
        }
      } else if (Rd == 2) {
        C v0 = *x0, v1 = *x1;
        C w1 = tw[k * tstep];
        if (sign > 0) w1.y = -w1.y;
        if constexpr (kF64) {
          tan_radix2(v0, v1, w1, *x0, *x1);
        } else {
          v1 = cmul(v1, w1);
          *x0 = mkc<C>(v0.x + v1.x, v0.y + v1.y);
          *x1 = mkc<C>(v0.x - v1.x, v0.y - v1.y);
        }
      } else {
        C *const x2 = a + i0 + 2 * p;
        C v0 = *x0, v1 = *x1, v2 = *x2;
        if (!kF64 || st > 0) {
          C w1 = tw[k * tstep], w2 = tw[2 * k * tstep];
          if (sign > 0) {
            w1.y = -w1.y;
            w2.y = -w2.y;
          }
          if constexpr (kF64) {
            v1 = tan_mul(v1, w1);
            v2 = tan_mul(v2, w2);
          } else {
            v1 = cmul(v1, w1);
            v2 = cmul(v2, w2);
          }
        }
        const R s3 = (R)0.86602540378443864676 * (R)sign;
        const C sm = mkc<C>(v1.x + v2.x, v1.y + v2.y), df = mkc<C>(v1.x - v2.x, v1.y - v2.y);
        if constexpr (kF64) {
          const C m1 = mkc<C>(fma(-0.5, sm.x, v0.x), fma(-0.5, sm.y, v0.y));
          *x0 = mkc<C>(v0.x + sm.x, v0.y + sm.y);
          *x1 = mkc<C>(fma(-s3, df.y, m1.x), fma(s3, df.x, m1.y));
          *x2 = mkc<C>(fma(s3, df.y, m1.x), fma(-s3, df.x, m1.y));
          continue;
        }
        const C m1 = mkc<C>(v0.x - (R)0.5 * sm.x, v0.y - (R)0.5 * sm.y);
        const C m2 = mkc<C>(-s3 * df.y, s3 * df.x);
        *x0 = mkc<C>(v0.x + sm.x, v0.y + sm.y);
        *x1 = mkc<C>(m1.x + m2.x, m1.y + m2.y);
        *x2 = mkc<C>(m1.x - m2.x, m1.y - m2.y);
      }
    }
    __syncthreads();
    p = q;
  }
}

}  // namespace
}  // namespace glass
