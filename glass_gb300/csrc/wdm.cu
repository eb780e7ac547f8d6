// WDM (Wilson-Daubechies-Meyer) wavelet transforms for sm_103a.
//
// Forward (utils/src/glass_wavelet.c:293-303 and :410-460): a real FFT of the
// ND = NF*NT samples, then for every layer m = 0..NF the NT-1 FFT bins around
// m NT/2, weighted by the Meyer window, inverse-FFT'd over NT points; the
// layer's NT coefficients are the real or imaginary parts by the parity of
// n + m (layout wdm[n + NT m], DC and Nyquist layers packed into row 0).
// Inverse (:351-405 and utils/src/glass_math.c:819-828): per layer an NT-point
// FFT of the coefficients, windowed overlap-add into the ND/2+1 bins, inverse
// real FFT.
//
// GPU structure:
//  * the real FFT of ND samples is a complex FFT of M = ND/2 packed samples
//    (x[2n] + i x[2n+1]), done four-step as M1 x M2: FFTs down the M2 columns
//    with the exp(-2 pi i n2 k1 / M) twiddle folded in, then FFTs along the M1
//    rows;
//  * one CTA per layer, or a cluster per pair of layers, for the windowed NT-point
//    transforms;
//  * grids of the form 2^a 3^b, so NF = 1536 (the reference's default grid) works.
//
// FP64 (parity with the reference) is bound by the FP64 pipe, so FP64
// instructions per sample are what counts, and warps enough to keep the pipe
// full:
//  * all FFTs run in place (fft_dit.cuh; twiddles from L1), 16 bytes of shared
//    memory per point instead of 48 with ping-pong buffers and a twiddle copy: 16
//    and more warps per SM instead of 8, which kept the pipe 65% busy;
//  * two layers share a transform.  Of a layer's inverse FFT each pixel uses the
//    real or the imaginary part; multiplied by (-i)^n (a shift of the spectrum by
//    NT/4) those are the real part, up to a sign s(n) of period four, so layers a
//    and b are the real and imaginary part of the inverse FFT of H_a + i H_b, H
//    the Hermitian parts.  The inverse runs the same backwards.  Only between a
//    series and its coefficients, where every value depends on all others: to and
//    from a spectrum a layer belongs to its own bins, and a transform shared with a
//    neighbour would give it rounding of that one's size, and its NaNs (a layer
//    beside one of 1e12 times its size lost all but four digits).  One layer per
//    transform there: 1024 x 2048 from a spectrum 192 us where pairs take 100,
//    1536 x 4096 to one 865 us where they take 331;
//  * the real spectrum is unpacked in the row pass and packed in the inverse's
//    column pass, where both bins k and M - k are at hand (one product for the two).
//  * the transforms' factors are in tangent form (fp64_math.cuh), those between
//    the passes in full tables;
//  * the pairs of layers and of rows are spread over clusters, as 385 or 513 equal
//    units leave a sixth of 152 SMs idle in the last wave.
// 107 -> 57 FP64 instructions per sample forward, 104 -> 60 inverse.  2^21 samples
// (1024 x 2048) forward 538 -> 245 us; 6.3 M samples (1536 x 4096) inverse 1787 ->
// 755 us.
//
// FP32 (GLASS_PREC_MIXED), and in FP64 the layers of the spectrum forms and of grids
// whose NT is not a multiple of 4, run one layer per CTA on ping-pong Stockham
// transforms; there the inverse's overlap-add runs in two launches (even, then odd
// layers: the supports of same-parity layers are disjoint, so no atomics are needed
// and the sum order is fixed).
#include <cooperative_groups.h>
#include <math.h>

#include <mutex>
#include <type_traits>
#include <vector>

#include "fft_dit.cuh"
#include "glass_common.cuh"
#include "wdm.cuh"

namespace glass {
namespace {

template <typename R>
struct Cx;
template <>
struct Cx<double> {
  using T = double2;
};
template <>
struct Cx<float> {
  using T = float2;
};

template <typename C>
__device__ __forceinline__ C cm(C a, C b) {
  C r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename C>
__device__ __forceinline__ C ca(C a, C b) {
  C r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}
template <typename C>
__device__ __forceinline__ C cs(C a, C b) {
  C r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}
template <typename C>
__device__ __forceinline__ C cconj(C a) {
  a.y = -a.y;
  return a;
}
template <typename C, typename R>
__device__ __forceinline__ C csc(C a, R s) {
  a.x *= s;
  a.y *= s;
  return a;
}
template <typename C>
__device__ __forceinline__ C mk(decltype(C().x) x, decltype(C().x) y) {
  C r;
  r.x = x;
  r.y = y;
  return r;
}

// e^{sign 2 pi i p / P} from two tables: lo[j] = e^{-2 pi i j/P} (j < K) and
// hi[j] = e^{-2 pi i j K/P}, p = hi K + lo.
template <typename C>
__device__ __forceinline__ C twiddle2(const C *lo, const C *hi, long long p, int K, int sign) {
  C t = cm(hi[p / K], lo[p % K]);
  return sign > 0 ? cconj(t) : t;
}

// In-place-looking mixed-radix Stockham FFT of nser series of length L stored
// series-major in a; b is a scratch buffer of the same size; tw[j] =
// exp(-2 pi i j / L).  All threads of the CTA take part.  Returns the buffer
// holding the result.  sign -1: forward, +1: inverse (unnormalised).
template <typename C>
__device__ C *block_fft(C *a, C *b, int L, int nser, const C *tw, int sign) {
  using R = decltype(C().x);
  int p = 1, rem = L;
  const R s3 = (R)0.86602540378443864676;  // sin(2 pi/3)
  while (rem > 1) {
    const int Rd = (rem % 3 == 0) ? 3 : (rem % 4 == 0) ? 4 : 2;
    const int nb = L / Rd;
    const int step = L / (p * Rd);
    for (int t = threadIdx.x; t < nser * nb; t += blockDim.x) {
      const int s = t / nb, i = t - s * nb;
      const int k = i % p;
      const C *src = a + (size_t)s * L;
      C *dst = b + (size_t)s * L;
      const int j = (i - k) * Rd + k;
      if (Rd == 4) {
        C v0 = src[i], v1 = src[i + nb], v2 = src[i + 2 * nb], v3 = src[i + 3 * nb];
        C w1 = tw[k * step], w2 = tw[2 * k * step], w3 = tw[3 * k * step];
        if (sign > 0) {
          w1 = cconj(w1);
          w2 = cconj(w2);
          w3 = cconj(w3);
        }
        v1 = cm(v1, w1);
        v2 = cm(v2, w2);
        v3 = cm(v3, w3);
        C t0 = ca(v0, v2), t1 = cs(v0, v2), t2 = ca(v1, v3), t3 = cs(v1, v3);
        // t3 * (-i sign): forward uses -i
        C t3r = sign < 0 ? mk<C>(t3.y, -t3.x) : mk<C>(-t3.y, t3.x);
        dst[j] = ca(t0, t2);
        dst[j + p] = ca(t1, t3r);
        dst[j + 2 * p] = cs(t0, t2);
        dst[j + 3 * p] = cs(t1, t3r);
      } else if (Rd == 2) {
        C v0 = src[i], v1 = src[i + nb];
        C w1 = tw[k * step];
        if (sign > 0) w1 = cconj(w1);
        v1 = cm(v1, w1);
        dst[j] = ca(v0, v1);
        dst[j + p] = cs(v0, v1);
      } else {
        C v0 = src[i], v1 = src[i + nb], v2 = src[i + 2 * nb];
        C w1 = tw[k * step], w2 = tw[2 * k * step];
        if (sign > 0) {
          w1 = cconj(w1);
          w2 = cconj(w2);
        }
        v1 = cm(v1, w1);
        v2 = cm(v2, w2);
        // radix-3 DFT with w = exp(sign 2 pi i / 3) = -1/2 + i sign sqrt(3)/2
        C sum = ca(v1, v2), dif = cs(v1, v2);
        C y0 = ca(v0, sum);
        C m1 = mk<C>(v0.x - (R)0.5 * sum.x, v0.y - (R)0.5 * sum.y);
        C m2 = mk<C>(-(R)sign * s3 * dif.y, (R)sign * s3 * dif.x);  // i sign sqrt3/2 dif
        dst[j] = y0;
        dst[j + p] = ca(m1, m2);
        dst[j + 2 * p] = cs(m1, m2);
      }
    }
    __syncthreads();
    C *tmp = a;
    a = b;
    b = tmp;
    p *= Rd;
    rem /= Rd;
  }
  return a;
}

template <typename C>
__device__ void load_twiddles(C *tw, const C *twg, int L) {
  for (int i = threadIdx.x; i < L; i += blockDim.x) tw[i] = twg[i];
}

// Four-step pass 1: FFTs of length M1 down ncol adjacent columns (stride M2)
// of src, times exp(sign 2 pi i n2 k1/M), written to dst at the same
// positions.  src may be the real input viewed as packed complex samples.
template <typename C>
__global__ void wdm_col_kernel(const C *src, C *dst, int M1, int M2, int ncol, const C *tw1, const C *tlo,
                               const C *thi, int K, int sign) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  C *tw = reinterpret_cast<C *>(sm_raw);
  C *a = tw + M1;
  C *b = a + (size_t)ncol * M1;
  load_twiddles(tw, tw1, M1);
  const int c0 = blockIdx.x * ncol;
  for (int t = threadIdx.x; t < ncol * M1; t += blockDim.x) {
    const int n1 = t / ncol, c = t - n1 * ncol;
    a[(size_t)c * M1 + n1] = src[(size_t)n1 * M2 + c0 + c];
  }
  __syncthreads();
  C *r = block_fft(a, b, M1, ncol, tw, sign);
  const long long M = (long long)M1 * M2;
  for (int t = threadIdx.x; t < ncol * M1; t += blockDim.x) {
    const int k1 = t / ncol, c = t - k1 * ncol;
    const long long p = ((long long)(c0 + c) * k1) % M;
    dst[(size_t)k1 * M2 + c0 + c] = cm(r[(size_t)c * M1 + k1], twiddle2(tlo, thi, p, K, sign));
  }
}

// Four-step pass 2: FFTs of length M2 along nrow rows of src; output index
// k1 + M1 k2 (natural order), times `scale`.
template <typename C>
__global__ void wdm_row_kernel(const C *src, C *dst, int M1, int M2, int nrow, const C *tw2, int sign,
                               decltype(C().x) scale) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  C *tw = reinterpret_cast<C *>(sm_raw);
  C *a = tw + M2;
  C *b = a + (size_t)nrow * M2;
  load_twiddles(tw, tw2, M2);
  const int r0 = blockIdx.x * nrow;
  for (int t = threadIdx.x; t < nrow * M2; t += blockDim.x) a[t] = src[(size_t)r0 * M2 + t];
  __syncthreads();
  C *r = block_fft(a, b, M2, nrow, tw, sign);
  for (int t = threadIdx.x; t < nrow * M2; t += blockDim.x) {
    const int rr = t / M2, k2 = t - rr * M2;
    dst[(size_t)(r0 + rr) + (size_t)M1 * k2] = csc(r[t], scale);
  }
}

// Bin k (0 <= k <= M) of the real spectrum of ND = 2M samples from the complex
// spectrum Z of the packed samples: X = (Z_k + Z*_{M-k})/2 - i e^{-2 pi i k/ND} (Z_k - Z*_{M-k})/2.
template <typename C>
__device__ __forceinline__ C real_bin(const C *Z, long long M, long long k, const C *tlo, const C *thi, int K) {
  using R = decltype(C().x);
  const C zk = Z[k % M], zm = cconj(Z[(M - k) % M]);
  const C e = twiddle2(tlo, thi, k, K, -1);  // e^{-2 pi i k/(2M)}
  const C s = ca(zk, zm), d = cs(zk, zm);
  const C ed = cm(e, d);
  return mk<C>((R)0.5 * (s.x + ed.y), (R)0.5 * (s.y - ed.x));
}

// Forward layers: one CTA per layer m in [0, NF].  X: the spectrum's bins 0..M times
// scale, or (PACKED) the FFT of the packed samples, unpacked on the fly with the
// tables tlo and thi.
template <typename C, bool PACKED>
__global__ void wdm_fwd_layer_kernel(const C *X, long long M, int NF, int NT,
                                     const decltype(C().x) *phif, const C *twNT, const C *tlo, const C *thi, int K,
                                     decltype(C().x) scale, decltype(C().x) *wdm) {
  using R = decltype(C().x);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  C *tw = reinterpret_cast<C *>(sm_raw);
  C *a = tw + NT;
  C *b = a + NT;
  load_twiddles(tw, twNT, NT);
  const int m = blockIdx.x;
  const int center = m * NT / 2;
  for (int t = threadIdx.x; t < NT; t += blockDim.x) {
    const int j = t - NT / 2;
    C v = mk<C>((R)0, (R)0);
    const int idx = center + j;
    bool ok = j > -NT / 2;
    if (m == 0 && idx < 0) ok = false;
    if (m == NF && idx > center) ok = false;
    if (ok) {
      R w = phif[j < 0 ? -j : j];
      if (j == 0 && (m == 0 || m == NF)) w *= (R)0.5;
      if constexpr (PACKED)
        v = csc(real_bin(X, M, (long long)idx, tlo, thi, K), w);
      else
        v = csc(X[idx], w);
    }
    a[t] = v;
  }
  __syncthreads();
  C *r = block_fft(a, b, NT, 1, tw, +1);
  const R inv = scale / (R)NT;  // scale 1 (FP32): exact
  const R sq2 = (R)1.41421356237309504880;
  for (int n = threadIdx.x; n < NT; n += blockDim.x) {
    const C v = r[n];
    if (m == 0) {
      if (!(n & 1)) wdm[n] = v.x * inv * sq2;
    } else if (m == NF) {
      if (!(n & 1)) wdm[n + 1] = v.x * inv * sq2;
    } else {
      const R sgn = (m % 2 == 0) ? (R)1 : (R)-1;
      wdm[n + (size_t)NT * m] = ((n + m) % 2 == 0) ? v.x * inv : sgn * v.y * inv;
    }
  }
}

// Inverse layers of one parity: X[i] += scale * window * FFT(prefactors) for the
// layer's support; layers m = parity, parity + 2, ...
template <typename C>
__global__ void wdm_inv_layer_kernel(const decltype(C().x) *wdm, int NF, int NT, int parity,
                                     const decltype(C().x) *phif, const C *twNT, decltype(C().x) scale, C *X) {
  using R = decltype(C().x);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  C *tw = reinterpret_cast<C *>(sm_raw);
  C *a = tw + NT;
  C *b = a + NT;
  load_twiddles(tw, twNT, NT);
  const int m = parity + 2 * blockIdx.x;
  if (m > NF) return;
  const R isq2 = (R)0.70710678118654752440;
  for (int n = threadIdx.x; n < NT; n += blockDim.x) {
    C v;
    if (m == 0) {
      v = mk<C>(wdm[(2 * n) % NT] * isq2, (R)0);
    } else if (m == NF) {
      v = mk<C>(wdm[(2 * n) % NT + 1] * isq2, (R)0);
    } else {
      const R w = wdm[n + (size_t)NT * m];
      v = ((n + m) % 2 == 0) ? mk<C>(w, (R)0) : mk<C>((R)0, -w);
    }
    a[n] = v;
  }
  __syncthreads();
  C *r = block_fft(a, b, NT, 1, tw, -1);
  const long long ND = (long long)NF * NT;
  const int center = m * NT / 2;
  int imin = center - NT / 2, imax = center + NT / 2;
  if (imin < 0) imin = 0;
  if (imax > ND / 2 + 1) imax = (int)(ND / 2 + 1);
  for (int i = imin + threadIdx.x; i < imax; i += blockDim.x) {
    const int iind = i > center ? i - center : center - i;
    const C v = (m == 0 || m == NF) ? r[(2 * i) % NT] : r[i % NT];
    const R w = phif[iind] * scale;
    C acc = X[i];
    acc.x += v.x * w;
    acc.y += v.y * w;
    X[i] = acc;
  }
}

// Complex spectrum of the packed samples from the real spectrum X (bins 0..M,
// the imaginary parts of bins 0 and M ignored as an inverse real FFT does):
// Z_k = (X_k + X*_{M-k}) + i e^{2 pi i k/ND} (X_k - X*_{M-k}).
template <typename C>
__global__ void wdm_pack_kernel(const C *X, long long M, const C *tlo, const C *thi, int K, C *Z) {
  using R = decltype(C().x);
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  C xk = X[k], xm = X[M - k];
  if (k == 0) {
    xk.y = (R)0;
    xm.y = (R)0;
  }
  xm = cconj(xm);
  const C s = ca(xk, xm), d = cs(xk, xm);
  const C e = twiddle2(tlo, thi, k, K, +1);
  const C ed = cm(e, d);
  Z[k] = mk<C>(s.x - ed.y, s.y + ed.x);
}

// ------------------------------------------------------------------ FP64
// The passes' factors in tangent form, laid out as the passes read them (so that a
// factor costs a coalesced load, where a product of two small tables costs 4 of a
// point's 36 FP64 instructions): colf[c][k1] = e^{-2 pi i c k1/M} between the
// four-step passes, packf[c][n1] and unpackf[r][k2] = e^{-2 pi i k/ND} of the bins k
// = n1 M2 + c and r + M1 k2 where the inverse packs and the forward unpacks the real
// spectrum.  32 bytes per complex point, kept with the plan.
__device__ __forceinline__ double2 conj_tan(double2 w) { return make_double2(w.x, -w.y); }
__device__ double2 tan_root(long long p, long long P) {  // e^{-2 pi i p / P}, 0 <= p < P
  // quadrant and octant in integers: the angle taken is at most pi/4
  const long long q = 4 * p / P, r = 4 * p - q * P;
  const bool flip = 2 * r > P;
  double s, c;
  sincospi(0.5 * ((double)(flip ? P - r : r) / (double)P), &s, &c);
  if (flip) {
    const double t = s;
    s = c;
    c = t;
  }
  return q == 0 ? tan_form(c, -s) : q == 1 ? tan_form(-s, -c) : q == 2 ? tan_form(-c, s) : tan_form(s, c);
}
__global__ void wdm_roots64_kernel(double2 *colf, double2 *packf, double2 *unpackf, int M1, int M2) {
  const long long M = (long long)M1 * M2, n1 = (long long)(M2 / 2 + 1) * M1, n2 = (long long)(M1 / 2 + 1) * M2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M + n1 + n2; i += (long long)gridDim.x * blockDim.x) {
    if (i < M)
      colf[i] = tan_root((i / M1) * (i % M1), M);
    else if (i < M + n1)
      packf[i - M] = tan_root(((i - M) % M1) * M2 + (i - M) / M1, 2 * M);
    else
      unpackf[i - M - n1] = tan_root((i - M - n1) / M2 + (i - M - n1) % M2 * M1, 2 * M);
  }
}

// Four-step pass 1, one column per CTA (16-byte accesses: two CTAs read each
// sector, which L2 serves; the FP64 pipe is the bound, and 1024 CTAs balance
// over 152 SMs where 256 of four columns leave a sixth of them idle).
__global__ void __launch_bounds__(256) wdm_col64_kernel(const double2 *src, double2 *dst, int M1, int M2,
                                                        const double2 *tw1, const double2 *colf) {
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  RadixPlan P;
  radix_plan(M1, P);
  const int c = blockIdx.x;
  for (int n1 = threadIdx.x; n1 < M1; n1 += blockDim.x) sm64[digit_rev(n1, P)] = src[(size_t)n1 * M2 + c];
  __syncthreads();
  dit_fft<-1>(sm64, M1, P, tw1, 1);
  for (int k1 = threadIdx.x; k1 < M1; k1 += blockDim.x)
    dst[(size_t)k1 * M2 + c] = tan_mul(sm64[k1], colf[(size_t)c * M1 + k1]);
}

// The inverse's pass 1 on columns c and M2 - c, whose elements are bins k and M -
// k of the real spectrum X (bins 0..M, the imaginary parts of bins 0 and M
// ignored as an inverse real FFT does): with s = X_k + X*_{M-k}, d = X_k - X*_{M-k}
// and w = e^{2 pi i k/ND} d, the packed spectrum is Z_k = s + i w, Z_{M-k} = s* + i w*.
__global__ void __launch_bounds__(512) wdm_pack_col64_kernel(const double2 *X, double2 *dst, int M1, int M2,
                                                             const double2 *tw1, const double2 *colf,
                                                             const double2 *packf) {
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  RadixPlan P;
  radix_plan(M1, P);
  const long long M = (long long)M1 * M2;
  const int c = blockIdx.x, cm = c == 0 ? 0 : M2 - c;
  const bool two = cm != c;
  const int bo = two ? M1 : 0;  // column M2 - c's place
  // column c's rows, each with its mirror: row M1 - n1 of column 0 (row 0 with bin
  // M), else row M1 - 1 - n1 of column M2 - c; a lone column's mirrors repeat it
  const int rows = two ? M1 : c == 0 ? M1 / 2 + 1 : (M1 + 1) / 2;
  for (int n1 = threadIdx.x; n1 < rows; n1 += blockDim.x) {
    const long long k = (long long)n1 * M2 + c;
    double2 xk = X[k], xm = X[M - k];
    if (k == 0) xk.y = xm.y = 0.0;
    const double2 s = make_double2(xk.x + xm.x, xk.y - xm.y), d = make_double2(xk.x - xm.x, xk.y + xm.y);
    const double2 w = tan_mul(d, conj_tan(packf[(size_t)c * M1 + n1]));
    sm64[digit_rev(n1, P)] = make_double2(s.x - w.y, s.y + w.x);
    if (k > 0) {
      const int nm = c == 0 ? M1 - n1 : M1 - 1 - n1;
      if (two || nm != n1) sm64[bo + digit_rev(nm, P)] = make_double2(s.x + w.y, w.x - s.y);
    }
  }
  __syncthreads();
  dit_fft<+1>(sm64, M1, P, tw1, 1, two ? 2 : 1);
  for (int t = threadIdx.x; t < (two ? 2 * M1 : M1); t += blockDim.x) {
    const int which = t >= M1, k1 = t - which * M1, col = which ? cm : c;
    dst[(size_t)k1 * M2 + col] = tan_mul(sm64[t], conj_tan(colf[(size_t)col * M1 + k1]));
  }
}

// The inverse's pass 2, one row per CTA: output index k1 + M1 k2.
__global__ void __launch_bounds__(256) wdm_row64_kernel(const double2 *src, double2 *dst, int M1, int M2,
                                                        const double2 *tw2) {
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  RadixPlan P;
  radix_plan(M2, P);
  const int r = blockIdx.x;
  for (int t = threadIdx.x; t < M2; t += blockDim.x) sm64[digit_rev(t, P)] = src[(size_t)r * M2 + t];
  __syncthreads();
  dit_fft<+1>(sm64, M2, P, tw2, 1);
  for (int k2 = threadIdx.x; k2 < M2; k2 += blockDim.x) dst[(size_t)r + (size_t)M1 * k2] = sm64[k2];
}

// The forward's pass 2 on rows k1 and M1 - k1, whose elements are bins k = k1 +
// M1 k2 and M - k of the packed spectrum Z, unpacked to twice the real spectrum:
// with s = Z_k + Z*_{M-k}, d = Z_k - Z*_{M-k} and w = e^{-2 pi i k/ND} d, 2 X_k = s - i w
// and 2 X_{M-k} = s* - i w*.
//
// A cluster of two CTAs per pair, a row each: 1026 CTAs balance over 152 SMs where
// 513 leave a sixth of them idle (88 -> 77 us at 1024 x 1024 points).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256) wdm_row_unpack64_kernel(const double2 *src, double2 *X,
                                                                                        int M1, int M2,
                                                                                        const double2 *tw2,
                                                                                        const double2 *unpackf) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  RadixPlan P;
  radix_plan(M2, P);
  const long long M = (long long)M1 * M2;
  const int h = (int)cluster.block_rank(), r = blockIdx.x >> 1, rm = r == 0 ? 0 : M1 - r;
  const bool two = rm != r;
  if (two || h == 0) {
    for (int k2 = threadIdx.x; k2 < M2; k2 += blockDim.x)
      sm64[digit_rev(k2, P)] = src[(size_t)(h ? rm : r) * M2 + k2];
    __syncthreads();
    dit_fft<-1>(sm64, M2, P, tw2, 1);
  }
  cluster.sync();  // both rows are transformed
  const double2 *Z = cluster.map_shared_rank(sm64, 0), *Zm = cluster.map_shared_rank(sm64, two ? 1 : 0);
  const int n = two ? M2 : r == 0 ? M2 / 2 + 1 : (M2 + 1) / 2;
  const int lo = h ? (n + 1) / 2 : 0, hi = h ? n : (n + 1) / 2;  // this CTA's part
  for (int k2 = lo + threadIdx.x; k2 < hi; k2 += blockDim.x) {
    const long long k = (long long)r + (long long)M1 * k2;
    const double2 zk = Z[k2], zm = Zm[r == 0 ? (k2 == 0 ? 0 : M2 - k2) : M2 - 1 - k2];
    const double2 s = make_double2(zk.x + zm.x, zk.y - zm.y), d = make_double2(zk.x - zm.x, zk.y + zm.y);
    const double2 w = tan_mul(d, unpackf[(size_t)r * M2 + k2]);
    X[k] = make_double2(s.x + w.y, s.y - w.x);
    if (2 * k != M) X[M - k] = make_double2(s.x - w.y, -(s.y + w.x));
  }
  cluster.sync();  // no CTA leaves while the other reads its row
}

// Layers of pair q: 0: the grid's first and last (0, NF); q >= 1: 2 q - 1 and 2 q
// (the second absent where it would be NF).
__host__ __device__ __forceinline__ int layer_pairs(int NF) { return 1 + NF / 2; }

// Forward layers, a pair per CTA, from scale times the real spectrum X (scale:
// what the window must be multiplied with, 1/NT and the Hermitian parts' half
// included).  The first and last layer use the real parts of even n alone, as
// they are (no shift).
//
// A cluster of two CTAs per pair: CTA h takes the elements of parity h, half the
// transform's length, and the last radix-2 stage, over half of the outputs each,
// reads both halves (for 513 pairs 112 -> 102 us: 1026 CTAs balance over the SMs).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256) wdm_fwd_pair64_kernel(const double2 *X, int NF, int NT,
                                                                                      const double *phif,
                                                                                      const double2 *twNT, double scale,
                                                                                      double *wdm) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  const int q = blockIdx.x >> 1, par = (int)cluster.block_rank(), h = NT / 2;
  RadixPlan P;
  radix_plan(h, P);
  const bool edge = q == 0;
  const int ma = edge ? 0 : 2 * q - 1, mb = edge ? NF : 2 * q;
  const bool has_b = edge || mb < NF;
  if (!edge && ma >= NF) return;
  if (edge) scale *= 1.41421356237309504880;
  auto bin = [&](int m, int k) {
    const int j = k - h;
    double2 v = make_double2(0.0, 0.0);
    if (j == -h || (m == 0 && j < 0) || (m == NF && j > 0)) return v;
    double w = scale * phif[j < 0 ? -j : j];
    if (edge && j == 0) w *= 0.5;
    v = X[(size_t)m * h + j];
    v = make_double2(v.x * w, v.y * w);
    return (!edge && (m & 1)) ? make_double2(-v.y, v.x) : v;
  };
  // e = 0 .. NT/2 gives the elements p and NT - p: of the layer pairs, p = e + 3 NT/4
  // (mod NT) up to NT/4 and p = e above; of the edge layers, p = e.  Those of this
  // CTA's parity: n1 up to NT/4, from e1, then the rest, from e2.
  const int e1 = edge ? par : (par + 3 * (NT / 4)) & 1, n1 = e1 > NT / 4 ? 0 : (NT / 4 - e1) / 2 + 1;
  const int e2 = NT / 4 + 1 + ((NT / 4 + 1 + par) & 1), n2 = e2 > h ? 0 : (h - e2) / 2 + 1;
  for (int i = threadIdx.x; i < n1 + n2; i += blockDim.x) {
    const int e = i < n1 ? e1 + 2 * i : e2 + 2 * (i - n1);
    int k, kp, p, pp;
    if (edge) {
      k = p = e;
      kp = pp = e == 0 ? 0 : NT - e;
    } else {
      k = e <= NT / 4 ? e : NT / 4 + e;
      kp = e <= NT / 4 ? h - k : 3 * h - k;
      p = k < NT / 4 ? k + 3 * (NT / 4) : k - NT / 4;
      pp = kp < NT / 4 ? kp + 3 * (NT / 4) : kp - NT / 4;
    }
    const double2 zero = make_double2(0.0, 0.0);
    const double2 a0 = bin(ma, k), a1 = bin(ma, kp), b0 = has_b ? bin(mb, k) : zero, b1 = has_b ? bin(mb, kp) : zero;
    const double ax = a0.x + a1.x, ay = a0.y - a1.y, bx = b0.x + b1.x, by = b0.y - b1.y;
    sm64[digit_rev(p >> 1, P)] = make_double2(ax - by, ay + bx);
    if (pp != p) sm64[digit_rev(pp >> 1, P)] = make_double2(ax + by, bx - ay);
  }
  __syncthreads();
  dit_fft<+1>(sm64, h, P, twNT, 2);
  cluster.sync();  // both halves are transformed
  const double2 *E = cluster.map_shared_rank(sm64, 0), *O = cluster.map_shared_rank(sm64, 1);
  for (int k = par * (h / 2) + threadIdx.x; k < (par + 1) * (h / 2); k += blockDim.x) {
    if (edge && (k & 1)) continue;  // even n alone
    double2 v[2];
    tan_radix2(E[k], O[k], conj_tan(twNT[k]), v[0], v[1]);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int n = k + u * h;
      if (edge) {
        wdm[n] = v[u].x;
        wdm[n + 1] = v[u].y;
      } else {
        wdm[n + (size_t)NT * ma] = (n & 2) ? -v[u].x : v[u].x;
        if (has_b) wdm[n + (size_t)NT * mb] = (n & 2) ? -v[u].y : v[u].y;
      }
    }
  }
  cluster.sync();  // no CTA leaves while the other reads its half
}

// Inverse layers, a pair per CTA: the FFT of u_a + i u_b, u a layer's coefficients
// with their signs, gives both layers' spectra, windowed and added into the bins
// of X.  No bin is cleared beforehand and the sum order is fixed: pairs 2q - 1, 2q
// reach bins [(q - 1) NT, (q + 1/2) NT); those of odd q store (first launch), those
// of even q add where a neighbour has stored and store between (second).  The
// first layer adds in the second launch; the last stores in the first where the
// pair below it is of even q, else adds in the second.  blockIdx: the launch's
// pairs, then its edge layers (first, last).
//
// A cluster of four CTAs per unit: CTA r takes the elements n = r (mod 4), a
// quarter of the transform's length, and the last radix-4 stage goes through
// distributed shared memory, every fourth butterfly each; then each forms a quarter
// of the bins (of 385 units 193 -> 159 us: 1540 CTAs balance over 152 SMs where
// 385 leave a sixth of the pipes idle).
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(256) wdm_inv_pair64_kernel(const double *wdm, int NF, int NT,
                                                                                      int launch, const double *phif,
                                                                                      const double2 *twNT, double scale,
                                                                                      double2 *X) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  grid_begin();
  extern __shared__ __align__(16) double2 sm64[];
  const int r = (int)cluster.block_rank(), unit = blockIdx.x >> 2, L = NT / 4;
  RadixPlan P;
  radix_plan(L, P);
  const int h = NT / 2, pairs = NF / 2, mine = launch == 0 ? (pairs + 1) / 2 : pairs / 2;
  const bool edge = unit >= mine;
  const int q = 2 * unit + 1 + launch;
  const int ma = 2 * q - 1, mb = 2 * q;
  const bool has_b = mb < NF;
  const bool last = edge && (launch == 0 || unit > mine);  // the edge CTA's layer is NF
  for (int n = r + 4 * threadIdx.x; n < NT; n += 4 * blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    if (edge) {
      v.x = wdm[(2 * n) % NT + last];
    } else {
      // layer a is odd, b even: the reference's (-i)^(n + m odd) as -i (-i)^n and
      // (-i)^n times these signs
      v.x = wdm[n + (size_t)NT * ma];
      if (has_b) v.y = wdm[n + (size_t)NT * mb];
      if ((n + 1) & 2) v.x = -v.x;
      if (n & 2) v.y = -v.y;
    }
    sm64[digit_rev(n >> 2, P)] = v;
  }
  __syncthreads();
  dit_fft<-1>(sm64, L, P, twNT, 4);
  cluster.sync();  // the four quarters are transformed
  double2 *S[4];
#pragma unroll
  for (int m = 0; m < 4; m++) S[m] = cluster.map_shared_rank(sm64, (unsigned)m);
  for (int k = r + 4 * threadIdx.x; k < L; k += 4 * blockDim.x) {
    double2 v0 = S[0][k], v1 = S[1][k], v2 = S[2][k], v3 = S[3][k];
    tan_radix4<-1>(v0, v1, v2, v3, twNT[k], twNT[2 * k]);
    S[0][k] = v0;
    S[1][k] = v1;
    S[2][k] = v2;
    S[3][k] = v3;
  }
  cluster.sync();  // bin k of the transform: S[k / L][k mod L]
  auto bin = [&](int k) {
    const int m = (k >= L) + (k >= 2 * L) + (k >= 3 * L);
    return cluster.map_shared_rank(sm64, (unsigned)m)[k - m * L];
  };
  if (edge) {
    const double c = scale * 0.70710678118654752440;
    const long long M = (long long)NF * h;
    // layer 0: bins 0 .. h - 1; layer NF: M - h .. M, bin M its own
    for (int i = r * blockDim.x + threadIdx.x; i < (last ? h + 1 : h); i += 4 * blockDim.x) {
      const long long k = last ? M - i : i;
      const double2 a = bin((int)((2 * k) % NT));
      const double w = c * phif[i];
      if (last && (i == 0 || launch == 0))
        X[k] = make_double2(w * a.x, w * a.y);
      else
        X[k] = make_double2(fma(w, a.x, X[k].x), fma(w, a.y, X[k].y));
    }
    cluster.sync();  // no CTA leaves while another reads its quarter
    return;
  }
  const double c = 0.5 * scale;
  // spectrum of layer a (real part's) or b at bin k of its own transform, twice
  auto part = [&](bool second, int k) {
    const double2 f = bin(k), g = bin(k == 0 ? 0 : NT - k);
    return second ? make_double2(f.y + g.y, g.x - f.x) : make_double2(f.x + g.x, f.y - g.y);
  };
  // bin i of layer m: R_m[i mod NT] = nu U_m[(i + NT/4) mod NT], nu = -i for layer a
  const int i0 = (q - 1) * NT, ca = ma * h, cb = ca + h;
  const int top = has_b ? NT : h;  // the upper layer's upper half
  for (int t = r * blockDim.x + threadIdx.x; t < top + h; t += 4 * blockDim.x) {
    const int i = i0 + t, k = (t + NT / 4) % NT;  // i0 is a multiple of NT
    double2 v = make_double2(0.0, 0.0);
    if (t < NT) {
      const double2 a = part(false, k);
      const double w = c * phif[i < ca ? ca - i : i - ca];
      v = make_double2(w * a.y, -(w * a.x));
    }
    if (has_b && t >= h) {
      const double2 b = part(true, k);
      const double w = c * phif[i < cb ? cb - i : i - cb];
      v = make_double2(fma(w, b.x, v.x), fma(w, b.y, v.y));
    }
    if (launch == 1 && (t < h || t >= top)) {  // the first launch has stored there
      const double2 x = X[i];
      v = make_double2(v.x + x.x, v.y + x.y);
    }
    X[i] = v;
  }
  cluster.sync();  // no CTA leaves while another reads its quarter
}

template <typename C>
__global__ void wdm_zero_kernel(C *X, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) X[i] = mk<C>((decltype(C().x))0, (decltype(C().x))0);
}

template <typename C>
__global__ void wdm_cast_kernel(const double *in, decltype(C().x) *out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (decltype(C().x))in[i];
}

template <typename C>
__global__ void wdm_uncast_kernel(const decltype(C().x) *in, double *out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (double)in[i];
}

}  // namespace

// ------------------------------------------------------------------ host side
static bool smooth23(long long x) {
  if (x <= 0) return false;
  while (x % 3 == 0) x /= 3;
  return (x & (x - 1)) == 0;
}

// M = M1 M2 with both factors of the form 2^a 3^b and at most maxL, as close
// to sqrt(M) as possible (balanced passes coalesce best).
static int split_factor(long long M, int maxL) {
  int best = 0;
  double bestd = 1e300;
  for (int L = 2; L <= maxL; L++) {
    if (M % L || !smooth23(L)) continue;
    const long long M2 = M / L;
    if (M2 < 2 || M2 > maxL || !smooth23(M2)) continue;
    const double d = fabs(log((double)L) - log((double)M2));
    if (d < bestd - 1e-12) {
      bestd = d;
      best = L;
    }
  }
  return best;
}

template <typename C>
static size_t fft_smem(int L, int nser) {
  return sizeof(C) * ((size_t)L + 2 * (size_t)nser * L);
}

constexpr int kMaxLine = 4096;                 // points of a row, column or layer
constexpr size_t kPassSmem = (size_t)200 << 10;  // of a pass of several series per CTA

// series per CTA for a pass over `count` series of length L
template <typename C>
static int pick_batch(int L, int count) {
  static_assert(sizeof(C) * 3 * kMaxLine <= kPassSmem, "one series fits");
  for (int n = 8; n > 1; n /= 2)
    if (count % n == 0 && fft_smem<C>(L, n) <= kPassSmem) return n;
  return 1;
}

// e^{-2 pi i j / P}: the angle is reduced to [0, pi] by conjugate symmetry
// before sin and cos are taken.
static void unit_root(long long j, long long P, double *c, double *s) {
  long long r = j % P;
  if (r < 0) r += P;
  double sg = -1.0;
  if (2 * r > P) {
    r = P - r;
    sg = 1.0;
  }
  const double a = 2.0 * M_PI * ((double)r / (double)P);
  *c = cos(a);
  *s = sg * sin(a);
}

template <typename C>
static void fill_roots(std::vector<C> &h, long long L) {
  h.resize((size_t)L);
  for (long long j = 0; j < L; j++) {
    double c, s;
    unit_root(j, L, &c, &s);
    h[(size_t)j].x = (decltype(C().x))c;
    h[(size_t)j].y = (decltype(C().x))s;
  }
}

// two-level table for e^{-2 pi i p / P}, p = hi K + lo
template <typename C>
static void fill_two_level(std::vector<C> &lo, std::vector<C> &hi, long long P, int K) {
  lo.resize(K);
  const long long nh = (P + K) / K;
  hi.resize((size_t)nh);
  for (int j = 0; j < K; j++) {
    double c, s;
    unit_root(j, P, &c, &s);
    lo[j].x = (decltype(C().x))c;
    lo[j].y = (decltype(C().x))s;
  }
  for (long long j = 0; j < nh; j++) {
    double c, s;
    unit_root(j * K, P, &c, &s);
    hi[(size_t)j].x = (decltype(C().x))c;
    hi[(size_t)j].y = (decltype(C().x))s;
  }
}

template <typename T>
static cudaError_t upload(void *dst, const std::vector<T> &v, cudaStream_t s) {
  return cudaMemcpyAsync(dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, s);
}

template <typename C>
static cudaError_t prepare_t(WdmPlan &P, int NF, int NT, const double *window, cudaStream_t s) {
  using R = decltype(C().x);
  const long long ND = (long long)NF * NT, M = ND / 2;
  P.NF = NF;
  P.NT = NT;
  P.M = M;
  P.M1 = split_factor(M, kMaxLine);
  if (!P.M1) return cudaErrorInvalidValue;
  P.M2 = (int)(M / P.M1);
  P.K = 1024;
  std::vector<C> t1, t2, tn, mlo, mhi, nlo, nhi;
  fill_roots(t1, P.M1);
  fill_roots(t2, P.M2);
  fill_roots(tn, NT);
  std::vector<C> ttn;
  if constexpr (sizeof(R) == 8) {  // dit_fft's; the wdm_*_layer_kernels take twNT as it is
    for (C &w : t1) w = tan_form(w.x, w.y);
    for (C &w : t2) w = tan_form(w.x, w.y);
    for (C w : tn) ttn.push_back(tan_form(w.x, w.y));
  }
  // FP32: two-level tables, and the four-step passes' and packed spectrum's buffer
  const size_t f32 = sizeof(R) == 4 ? sizeof(C) : 0;
  if (f32) {
    fill_two_level(mlo, mhi, M, P.K);
    fill_two_level(nlo, nhi, ND, P.K);
  }
  std::vector<R> win(NT / 2 + 1);
  for (int i = 0; i <= NT / 2; i++) win[i] = (R)window[i];
  const size_t elem = sizeof(C);
  auto pad = [](size_t n) { return (n + 255) / 256 * 256; };
  // FP64: the passes' factors (wdm_roots64_kernel)
  const size_t full = sizeof(R) == 8 ? elem : 0;
  const size_t sizes[16] = {elem * t1.size(), elem * t2.size(), elem * tn.size(), elem * mlo.size(),
                            elem * mhi.size(), elem * nlo.size(), elem * nhi.size(), sizeof(R) * win.size(),
                            f32 * (size_t)(M + 1), elem * (size_t)(M + 1), elem * (size_t)(M + 1),
                            sizeof(double) * (size_t)ND,
                            full * (size_t)M, full * (size_t)(P.M2 / 2 + 1) * P.M1, full * (size_t)(P.M1 / 2 + 1) * P.M2,
                            elem * ttn.size()};
  size_t bytes = 0;
  for (size_t b : sizes) bytes += pad(b);
  cudaError_t e = cudaMalloc(&P.base, bytes);
  if (e != cudaSuccess) {
    P.base = nullptr;
    return e;
  }
  void **slots[16] = {&P.tw1, &P.tw2, &P.twNT, &P.mlo,  &P.mhi,  &P.nlo,   &P.nhi,    &P.win,
                      &P.bufA, &P.bufB, &P.bufX, &P.rbuf, &P.colf, &P.packf, &P.unpackf,
                      &P.ttNT};
  char *p = (char *)P.base;
  for (int i = 0; i < 16; i++) {
    *slots[i] = p;
    p += pad(sizes[i]);
  }
  if ((e = upload(P.tw1, t1, s)) != cudaSuccess) return e;
  if ((e = upload(P.tw2, t2, s)) != cudaSuccess) return e;
  if ((e = upload(P.twNT, tn, s)) != cudaSuccess) return e;
  if ((e = upload(P.win, win, s)) != cudaSuccess) return e;
  if constexpr (sizeof(R) == 4) {
    if ((e = upload(P.mlo, mlo, s)) != cudaSuccess) return e;
    if ((e = upload(P.mhi, mhi, s)) != cudaSuccess) return e;
    if ((e = upload(P.nlo, nlo, s)) != cudaSuccess) return e;
    if ((e = upload(P.nhi, nhi, s)) != cudaSuccess) return e;
  } else {
    if ((e = upload(P.ttNT, ttn, s)) != cudaSuccess) return e;
    wdm_roots64_kernel<<<1024, 256, 0, s>>>((double2 *)P.colf, (double2 *)P.packf, (double2 *)P.unpackf, P.M1, P.M2);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaStreamSynchronize(s);  // the host vectors go out of scope
}

// Complex FFT of M = M1 x M2 points, src -> dst (natural order), four-step.
template <typename C>
static cudaError_t four_step(const WdmPlan &P, const C *src, C *tmp, C *dst, int sign, decltype(C().x) scale,
                             cudaStream_t s) {
  const int M1 = P.M1, M2 = P.M2;
  const int nc = pick_batch<C>(M1, M2), nr = pick_batch<C>(M2, M1);
  const size_t sm1 = fft_smem<C>(M1, nc), sm2 = fft_smem<C>(M2, nr);
  cudaError_t e;
  if ((e = smem_limit<wdm_col_kernel<C>>(kPassSmem)) != cudaSuccess) return e;
  if ((e = smem_limit<wdm_row_kernel<C>>(kPassSmem)) != cudaSuccess) return e;
  wdm_col_kernel<C><<<M2 / nc, 256, sm1, s>>>(src, tmp, M1, M2, nc, (const C *)P.tw1, (const C *)P.mlo,
                                               (const C *)P.mhi, P.K, sign);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  wdm_row_kernel<C><<<M1 / nr, 256, sm2, s>>>(tmp, dst, M1, M2, nr, (const C *)P.tw2, sign, scale);
  return cudaGetLastError();
}

static unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }

// ---- FP64
static size_t smem64(int points) { return sizeof(double2) * (size_t)points; }
static int threads64(int points, int most) {  // one radix-4 butterfly per thread
  int t = (points / 4 + 31) / 32 * 32;
  return t < 32 ? 32 : t > most ? most : t;
}
// most_points, most_threads: the most that any grid takes of the kernel.
template <auto K, typename... Args>
static cudaError_t launch64(int grid, int points, int most_points, int most_threads, cudaStream_t s, Args... args) {
  cudaError_t e;
  if (smem64(most_points) > 48 * 1024 && (e = smem_limit<K>(smem64(most_points))) != cudaSuccess) return e;
  return launch_chained(K, grid, threads64(points, most_threads), smem64(points), s, args...);
}

// Two layers to a transform: where all values depend on each other, and NT is a
// multiple of 4.
enum class Layers { kPaired, kSeparate };

// scale times the real spectrum X -> coefficients.
static cudaError_t fwd_layers64(const WdmPlan &P, Layers how, const double2 *X, double scale, double *wdm,
                                cudaStream_t s) {
  const int NF = P.NF, NT = P.NT;
  if (how == Layers::kPaired && NT % 4 == 0)
    return launch64<wdm_fwd_pair64_kernel>(2 * layer_pairs(NF), NT / 2, kMaxLine / 2, 256, s, X, NF, NT, (const double *)P.win,
                    (const double2 *)P.ttNT, 0.5 * scale / NT, wdm);
  const size_t sm = fft_smem<double2>(NT, 1);
  const cudaError_t e = smem_limit<wdm_fwd_layer_kernel<double2, false>>(fft_smem<double2>(kMaxLine, 1));
  if (e != cudaSuccess) return e;
  wdm_fwd_layer_kernel<double2, false><<<NF + 1, 256, sm, s>>>(
      X, P.M, NF, NT, (const double *)P.win, (const double2 *)P.twNT, nullptr, nullptr, 0, scale, wdm);
  return cudaGetLastError();
}

static cudaError_t forward64(const WdmPlan &P, const double *time, double *wdm, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT;
  const double2 *packed = reinterpret_cast<const double2 *>(time);
  cudaError_t e;
  if ((uintptr_t)time % 16) {  // the packed complex view needs 16-byte alignment
    if ((e = cudaMemcpyAsync(P.rbuf, time, sizeof(double) * ND, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
    packed = reinterpret_cast<const double2 *>(P.rbuf);
  }
  if ((e = launch64<wdm_col64_kernel>(P.M2, P.M1, kMaxLine, 256, s, packed, (double2 *)P.bufB, P.M1, P.M2,
                    (const double2 *)P.tw1, (const double2 *)P.colf)) != cudaSuccess)
    return e;
  if ((e = launch64<wdm_row_unpack64_kernel>(2 * (P.M1 / 2 + 1), P.M2, kMaxLine, 256, s, (const double2 *)P.bufB,
                    (double2 *)P.bufX, P.M1, P.M2, (const double2 *)P.tw2, (const double2 *)P.unpackf)) != cudaSuccess)
    return e;
  return fwd_layers64(P, Layers::kPaired, (const double2 *)P.bufX, 0.5, wdm, s);
}

// WDM -> scale times the spectrum, bins 0..M of P.bufX.
static cudaError_t inverse_layers64(const WdmPlan &P, Layers how, const double *wdm, double scale, cudaStream_t s) {
  const int NF = P.NF, NT = P.NT;
  const double *win = (const double *)P.win;
  double2 *X = (double2 *)P.bufX;
  cudaError_t e;
  scale *= 0.5 * NF;
  if (how == Layers::kPaired && NT % 4 == 0) {
    const double2 *tw = (const double2 *)P.ttNT;
    const int pairs = NF / 2;  // (1, 2), (3, 4), ...
    const bool last_first = pairs % 2 == 0;  // the last layer's place: see the kernel
    if ((e = launch64<wdm_inv_pair64_kernel>(4 * ((pairs + 1) / 2 + last_first), NT / 4, kMaxLine / 4, 256, s, wdm, NF, NT, 0, win,
                                             tw, scale, X)) != cudaSuccess)
      return e;
    return launch64<wdm_inv_pair64_kernel>(4 * (pairs / 2 + 1 + !last_first), NT / 4, kMaxLine / 4, 256, s, wdm, NF, NT, 1, win,
                                           tw, scale, X);
  }
  wdm_zero_kernel<double2><<<blocks_for(P.M + 1), 256, 0, s>>>(X, P.M + 1);
  const size_t sm = fft_smem<double2>(NT, 1);
  if ((e = smem_limit<wdm_inv_layer_kernel<double2>>(fft_smem<double2>(kMaxLine, 1))) != cudaSuccess) return e;
  for (int parity = 0; parity < 2; parity++)
    wdm_inv_layer_kernel<double2><<<(NF - parity) / 2 + 1, 256, sm, s>>>(wdm, NF, NT, parity, win, (const double2 *)P.twNT,
                                                                         scale, X);
  return cudaGetLastError();
}

static cudaError_t inverse64(const WdmPlan &P, const double *wdm, double *time, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT;
  cudaError_t e;
  if ((e = inverse_layers64(P, Layers::kPaired, wdm, 1.0 / (double)ND, s)) != cudaSuccess) return e;
  if ((e = launch64<wdm_pack_col64_kernel>(P.M2 / 2 + 1, 2 * P.M1, 2 * kMaxLine, 512, s, (const double2 *)P.bufX,
                    (double2 *)P.bufB, P.M1, P.M2, (const double2 *)P.tw1, (const double2 *)P.colf,
                    (const double2 *)P.packf)) != cudaSuccess)
    return e;
  const bool direct = (uintptr_t)time % 16 == 0;
  double2 *dst = reinterpret_cast<double2 *>(direct ? (void *)time : P.rbuf);
  if ((e = launch64<wdm_row64_kernel>(P.M1, P.M2, kMaxLine, 256, s, (const double2 *)P.bufB, dst, P.M1, P.M2,
                    (const double2 *)P.tw2)) != cudaSuccess)
    return e;
  if (!direct) return cudaMemcpyAsync(time, P.rbuf, sizeof(double) * ND, cudaMemcpyDeviceToDevice, s);
  return cudaSuccess;
}

// wdm -> ND/2 + 1 complex bins (ND + 2 doubles), wavelet_transform_inverse_freq
static cudaError_t to_freq64(const WdmPlan &P, const double *wdm, double *freq, cudaStream_t s) {
  const cudaError_t e = inverse_layers64(P, Layers::kSeparate, wdm, 1.0, s);
  if (e != cudaSuccess) return e;
  return cudaMemcpyAsync(freq, P.bufX, sizeof(double2) * (size_t)(P.M + 1), cudaMemcpyDeviceToDevice, s);
}

// ND/2 + 1 complex bins -> wdm, wavelet_transform_freq
static cudaError_t from_freq64(const WdmPlan &P, const double *freq, double *wdm, cudaStream_t s) {
  const double2 *X = reinterpret_cast<const double2 *>(freq);
  if ((uintptr_t)freq % 16) {
    const cudaError_t e =
        cudaMemcpyAsync(P.bufX, freq, sizeof(double2) * (size_t)(P.M + 1), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    X = (const double2 *)P.bufX;
  }
  return fwd_layers64(P, Layers::kSeparate, X, 1.0, wdm, s);
}

// ---- FP32 (double at the boundary)
static cudaError_t forward32(const WdmPlan &P, const double *time, double *wdm, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT;
  cudaError_t e;
  float *out = (float *)P.rbuf;  // consumed by the first FFT pass before the layers write
  wdm_cast_kernel<float2><<<blocks_for(ND), 256, 0, s>>>(time, out, ND);
  if ((e = four_step<float2>(P, (const float2 *)P.rbuf, (float2 *)P.bufB, (float2 *)P.bufA, -1, 1.f, s)) != cudaSuccess)
    return e;
  const size_t sm = fft_smem<float2>(P.NT, 1);
  if ((e = smem_limit<wdm_fwd_layer_kernel<float2, true>>(fft_smem<float2>(kMaxLine, 1))) != cudaSuccess) return e;
  wdm_fwd_layer_kernel<float2, true><<<P.NF + 1, 256, sm, s>>>(
      (const float2 *)P.bufA, P.M, P.NF, P.NT, (const float *)P.win, (const float2 *)P.twNT, (const float2 *)P.nlo,
      (const float2 *)P.nhi, P.K, 1.f, out);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  wdm_uncast_kernel<float2><<<blocks_for(ND), 256, 0, s>>>(out, wdm, ND);
  return cudaGetLastError();
}

// WDM -> spectrum: bins 0..M summed into P.bufX by the windowed layer transforms.
static cudaError_t inverse_layers32(const WdmPlan &P, const double *wdm, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT;
  const int NT = P.NT, NF = P.NF;
  wdm_cast_kernel<float2><<<blocks_for(ND), 256, 0, s>>>(wdm, (float *)P.rbuf, ND);
  wdm_zero_kernel<float2><<<blocks_for(P.M + 1), 256, 0, s>>>((float2 *)P.bufX, P.M + 1);
  const size_t sm = fft_smem<float2>(NT, 1);
  const cudaError_t e = smem_limit<wdm_inv_layer_kernel<float2>>(fft_smem<float2>(kMaxLine, 1));
  if (e != cudaSuccess) return e;
  // even layers, then odd: same-parity layers have disjoint supports
  for (int parity = 0; parity < 2; parity++)
    wdm_inv_layer_kernel<float2><<<(NF - parity) / 2 + 1, 256, sm, s>>>((const float *)P.rbuf, NF, NT, parity,
                                                                        (const float *)P.win, (const float2 *)P.twNT,
                                                                        (float)NF / 2.f, (float2 *)P.bufX);
  return cudaGetLastError();
}

static cudaError_t inverse32(const WdmPlan &P, const double *wdm, double *time, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT, M = P.M;
  cudaError_t e;
  if ((e = inverse_layers32(P, wdm, s)) != cudaSuccess) return e;
  wdm_pack_kernel<float2><<<blocks_for(M), 256, 0, s>>>((const float2 *)P.bufX, M, (const float2 *)P.nlo,
                                                        (const float2 *)P.nhi, P.K, (float2 *)P.bufA);
  if ((e = four_step<float2>(P, (const float2 *)P.bufA, (float2 *)P.bufB, (float2 *)P.rbuf, +1,
                             (float)(1.0 / (double)ND), s)) != cudaSuccess)
    return e;
  wdm_uncast_kernel<float2><<<blocks_for(ND), 256, 0, s>>>((const float *)P.rbuf, time, ND);
  return cudaGetLastError();
}

static cudaError_t to_freq32(const WdmPlan &P, const double *wdm, double *freq, cudaStream_t s) {
  const long long n = 2 * (P.M + 1);
  const cudaError_t e = inverse_layers32(P, wdm, s);
  if (e != cudaSuccess) return e;
  wdm_uncast_kernel<float2><<<blocks_for(n), 256, 0, s>>>((const float *)P.bufX, freq, n);
  return cudaGetLastError();
}

static cudaError_t from_freq32(const WdmPlan &P, const double *freq, double *wdm, cudaStream_t s) {
  const long long ND = (long long)P.NF * P.NT, n = 2 * (P.M + 1);
  wdm_cast_kernel<float2><<<blocks_for(n), 256, 0, s>>>(freq, (float *)P.bufX, n);
  const size_t sm = fft_smem<float2>(P.NT, 1);
  cudaError_t e = smem_limit<wdm_fwd_layer_kernel<float2, false>>(fft_smem<float2>(kMaxLine, 1));
  if (e != cudaSuccess) return e;
  wdm_fwd_layer_kernel<float2, false><<<P.NF + 1, 256, sm, s>>>((const float2 *)P.bufX, P.M, P.NF, P.NT,
                                                                (const float *)P.win, (const float2 *)P.twNT, nullptr,
                                                                nullptr, 0, 1.f, (float *)P.rbuf);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  wdm_uncast_kernel<float2><<<blocks_for(ND), 256, 0, s>>>((const float *)P.rbuf, wdm, ND);
  return cudaGetLastError();
}

bool wdm_grid_supported(int NF, int NT) {
  if (NF < 2 || NT < 8 || NT > kMaxLine || NT % 2 || !smooth23(NT)) return false;
  const long long M = (long long)NF * NT / 2;
  return split_factor(M, kMaxLine) != 0;
}

cudaError_t wdm_prepare(WdmPlan &P, int precision, int NF, int NT, const double *window, cudaStream_t s) {
  wdm_release(P);
  if (!wdm_grid_supported(NF, NT)) return cudaErrorInvalidValue;
  P.precision = precision;
  const cudaError_t e =
      precision == 1 ? prepare_t<float2>(P, NF, NT, window, s) : prepare_t<double2>(P, NF, NT, window, s);
  if (e != cudaSuccess) wdm_release(P);
  return e;
}

void wdm_release(WdmPlan &P) {
  if (P.base) cudaFree(P.base);
  P = WdmPlan();
}

cudaError_t wdm_forward(const WdmPlan &P, const double *time, double *wdm, cudaStream_t s) {
  return P.precision == 1 ? forward32(P, time, wdm, s) : forward64(P, time, wdm, s);
}

cudaError_t wdm_inverse(const WdmPlan &P, const double *wdm, double *time, cudaStream_t s) {
  return P.precision == 1 ? inverse32(P, wdm, time, s) : inverse64(P, wdm, time, s);
}

cudaError_t wdm_to_freq(const WdmPlan &P, const double *wdm, double *freq, cudaStream_t s) {
  return P.precision == 1 ? to_freq32(P, wdm, freq, s) : to_freq64(P, wdm, freq, s);
}

cudaError_t wdm_from_freq(const WdmPlan &P, const double *freq, double *wdm, cudaStream_t s) {
  return P.precision == 1 ? from_freq32(P, freq, wdm, s) : from_freq64(P, freq, wdm, s);
}

// Meyer window of utils/src/glass_wavelet.c:305-349 with the regularised
// incomplete beta function I_x(nx, nx) of utils/src/glass_math.c:1214-1242
// (hypergeometric series, which terminates for integer nx).
static double hyp2f1_series(double a, double b, double c, double x) {
  const double TOL = 1e-8;
  double term = a * b * x / c, value = 1.0 + term;
  int n = 1;
  while (fabs(term) > TOL) {
    a++, b++, c++, n++;
    term *= a * b * x / c / n;
    value += term;
  }
  return value;
}

void wdm_window(int NF, int NT, double A, double nx, bool forward, double *phif) {
  const double DeltaOmega = M_PI / NF, domega = 2 * DeltaOmega / (double)NT;
  const double B = DeltaOmega - 2 * A, insDOM = 1.0 / sqrt(DeltaOmega);
  const double beta = exp(lgamma(nx) + lgamma(nx) - lgamma(nx + nx));
  for (int i = 0; i < NT / 2 + 1; i++) {
    const double omega = domega * i;
    double z = 0.0;
    if (fabs(omega) >= A && fabs(omega) < A + B) {
      const double x = (fabs(omega) - A) / B;
      const double y = pow(x, nx) * hyp2f1_series(nx, 1 - nx, nx + 1, x) / beta / nx;
      z = insDOM * cos(y * M_PI_2);
    }
    if (fabs(omega) < A) z = insDOM;
    phif[i] = z;
  }
  double norm = 0.0;
  for (int i = 0; i < NT / 2 + 1; i++) norm += (i == 0 ? 1.0 : 2.0) * phif[i] * phif[i];
  norm = sqrt(norm * domega * M_1_PI);
  if (forward) norm *= NF / 2.0;
  for (int i = 0; i < NT / 2 + 1; i++) phif[i] /= norm;
}

}  // namespace glass
