// Noise-model likelihood of XYZ frequency-domain data for sm_103a: the noise
// module's instrument covariance (noise/src/glass_noise_model.c:389-546),
// optionally plus the galactic foreground (:612-654, added as
// generate_full_covariance_matrix does, :894-907), the 3x3 inverse and
// log-determinant (utils/src/glass_math.c:240-289) and my_noise_log_likelihood
// (noise/src/glass_noise_model.c:1243-1273), for a batch of noise models,
// optionally with a stochastic background (SGWB) of one of the reference's
// three spectral templates times the instrument's response
// (generate_sgwb_model, :778-842; the wavelet form :843-892).
//
// The reference regenerates the whole covariance, inverts it and sums the
// likelihood for every proposed noise model (noise_instrument_model_mcmc and
// noise_foreground_model_mcmc, noise/src/glass_noise_sampler.c:395-752), ten
// proposals per chain per sweep.  Everything that depends on frequency alone
// (the TDI and arm transfer functions, f^(-7/3), the data's auto- and
// cross-spectra) is tabulated once per bin when the data are set; a batch then
// costs one pass over the table per model.
//
// FP64.  The FP64 pipe bounds every kernel here (2 multiply-adds per SM and
// clock, 1/64 of FP32), so the FP64 instructions per model and bin are what is
// counted; integer work and loads are free beside them:
//  * the levels enter through 15 sums per model and five products of transfer
//    functions per bin (15 operations for the six covariance entries);
//  * the inverse is the cofactors over the determinant, with one reciprocal
//    (the reference takes exp(log|cofactor| - log det): the same numbers to a
//    few ulp of the covariance's conditioning);
//  * the log-determinants are summed as the product of their mantissas and the
//    sum of their exponents, one log per warp;
//  * the foreground's tanh is 1 / (1 + exp(2 (f - fk) / f2)), whose exponential
//    is a geometric sequence along a thread's bins, and its power law
//    exp(alpha (log f - log f1)) with log f tabulated.
// 420 -> 85 FP64 instructions per model and bin with the foreground; 1024
// models on 15360 bins 12.44 -> 2.45 ms, wavelet cells 202 -> 35 and 22.7 ->
// 3.56 ms (1024 models, 58880 cells, modulated foreground).  Compiled without
// multiply-add contraction (the SGWB templates keep the reference's operation
// order); the code below writes its multiply-adds out.

#include <math.h>

#include <vector>

#include "../../include/glass_gb300.h"
#include "fp64_math.cuh"
#include "glass_common.cuh"
#include "noise.cuh"

namespace glass {

namespace {

constexpr int kNoiseThreads = 128;
// Bins per thread of the Fourier kernels.  The most that still gives every SM
// a few CTAs, so that one model on a few thousand bins uses the whole chip (a
// warp's FP64 instruction holds its SM's pipe for 16 clocks: 2048 bins on one
// SM take 16x what they take on 16); at the most, a CTA's model constants and
// its reduction are 2% of its work.
constexpr int kNoiseMaxBins = 16;
constexpr int kNoiseCtasPerSm = 4;  // (608 on 152 SMs)

struct NoiseArgs {
  int N, nchunks, nprop, R;  // R bins per thread
  double fstep;              // 128 bins, in Hz
  const double *tab;  // kNoiseTabRows rows of N
  const double *inst;  // [nprop][12]
  const double *sgal;  // [nprop][5] or null
  int sg_type;         // SGWB template
  const double *sgwb;  // [nprop][4] or null
  const double *rsg;   // SGWB response, 6 rows of N
  double *partial;     // [nprop][nchunks]
};

// A sum of logarithms of positive normal numbers as the product of their
// mantissas, kept in [1, 2), and the sum of their exponents.
struct LogSum {
  double m = 1.0;
  int e = 0;
};
__device__ __forceinline__ double mantissa(double x, int &e) {
  const int hi = __double2hiint(x);
  e += (hi >> 20) - 1023;
  return __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
}
__device__ __forceinline__ void log_add(LogSum &s, double x) {
  const double m = mantissa(x, s.e);
  s.m = mantissa(s.m * m, s.e);
}
// Positive, finite and 2^-959 < x < 2^961: rcp_fast and log_add apply.
__device__ __forceinline__ bool plain_positive(double x) {
  return (unsigned)(__double2hiint(x) - 0x04000000) < 0x78000000u;
}

// The CTA's sum of chi and of the logarithms (valid in thread 0).
__device__ __forceinline__ double block_total(double chi, LogSum ld) {
  __shared__ double red[kNoiseThreads / 32], redm[kNoiseThreads / 32];
  __shared__ int rede[kNoiseThreads / 32];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    chi += __shfl_xor_sync(0xffffffffu, chi, off);
    ld.m *= __shfl_xor_sync(0xffffffffu, ld.m, off);  // below 2^32
  }
  ld.e = __reduce_add_sync(0xffffffffu, ld.e);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red[warp] = chi;
    redm[warp] = ld.m;
    rede[warp] = ld.e;
  }
  __syncthreads();
  double s = 0.0;
  if (warp == 0) {
    if (lane < kNoiseThreads / 32) s = red[lane] + fma((double)rede[lane], 0.693147180559945309417, log(redm[lane]));
#pragma unroll
    for (int off = kNoiseThreads / 64; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  }
  return s;
}

// ------------------------------------------------------ one model's constants
// The sums of link levels that the covariance entries use
// (noise/src/glass_noise_model.c:445-546): per diagonal entry xx, yy, zz the
// metrology sum o / 4 and the acceleration sums a and b (b times cos^2), per
// off-diagonal entry xy, xz, yz the metrology sum p / 2 and the acceleration
// sum 2 q; and the foreground's parameters (map_array_to_foreground_params,
// :67-74).
struct NoiseModel {
  double lev[15];  // o, a, b, p, q: three each
  double Amp, l1, alpha, fk, i2, f10, estep;
  int chain;  // the foreground's exponential may run as a geometric sequence
};
// Level indices of each sum in o, a, b, p, q (12: none), levels in the order
// 12, 21, 23, 32, 13, 31 (acceleration, then metrology).
__constant__ unsigned char kLevelIdx[15][4] = {
    {6, 7, 10, 11}, {8, 9, 7, 6},   {11, 10, 9, 8},  {0, 4, 12, 12}, {2, 1, 12, 12},
    {5, 3, 12, 12}, {1, 5, 12, 12}, {3, 0, 12, 12},  {4, 2, 12, 12}, {6, 7, 12, 12},
    {10, 11, 12, 12}, {9, 8, 12, 12}, {0, 1, 12, 12}, {4, 5, 12, 12}, {3, 2, 12, 12}};

// By the CTA's first warp, the foreground by its second; the caller synchronises.
// fstep: the frequency step between a thread's bins.
__device__ __forceinline__ void noise_foreground_load(NoiseModel &M, const double *sg, double fstep) {
  const int lane = threadIdx.x & 31;
  const double v = lane < 5 ? sg[lane] : 0.0, x = lane == 2 ? 0.0 : v;
  const double e = exp(x);
  const double f2 = __shfl_sync(0xffffffffu, e, 4);
  if (lane == 0) M.Amp = e;
  if (lane == 1) {
    M.l1 = v;
    M.f10 = e * 10;
  }
  if (lane == 2) M.alpha = v;
  if (lane == 3) M.fk = e;
  if (lane == 4) {
    // a step of the sequence by more than e^1 could leave the exponent range
    // within a thread's bins and not come back
    const double st = 2.0 * fstep / f2;
    M.i2 = 2.0 / f2;
    M.estep = exp(st);
    M.chain = st < 1.0;
  }
}

// At low frequencies the acceleration noise of X + Y + Z cancels to (1 - cos)^2 ~ 1e-7
// of its terms, for a (12 + 13, 23 + 21, 31 + 32), b (21 + 31, 32 + 12, 13 + 23) and
// s = q / 2 (12 + 21, 13 + 31, 23 + 32) that obey a_x + b_x = s_xy + s_xz and so on.
// Sums rounded one by one do so only to 1e-16, the same way in every bin, and
// the errors of the bins add up.  With s and a rounded to 50 bits of the largest s,
// b = s + s - a is exact: a model whose levels differ by 1e-15 of the largest.  Data that
// the model does not describe, 4000 bins from 0.1 mHz, link levels a factor of 2 apart: rms error
// of the likelihood against 80 bits 1.1e-10 -> 1.2e-11 (sums by bin, as the reference: 1.1e-11).
__device__ __forceinline__ void noise_model_load(NoiseModel &M, const double *in, const double *sg, double fstep) {
  if (threadIdx.x >= 64) return;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) {
    if (sg) noise_foreground_load(M, sg, fstep);
    return;
  }
  double lev = 0.0;
  if (lane < 15) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int i = kLevelIdx[lane][k];
      s += i < 12 ? in[i] : 0.0;
    }
    lev = s;
  }
  // the largest exponent of s (lanes 12 .. 14: xy, xz, yz); levels at the ends of the
  // range, and not finite ones, as they are
  const int ex = (__double2hiint(lev) >> 20) & 0x7ff;
  const int e = max(__shfl_sync(0xffffffffu, ex, 12), max(__shfl_sync(0xffffffffu, ex, 13), __shfl_sync(0xffffffffu, ex, 14)));
  if (e - 64u < 1900u) {
    const double R = __hiloint2double(((e + 3) << 20) | 0x80000, 0);  // adding 1.5 2^(e+3) rounds to 50 bits of 2^e
    if ((lane >= 3 && lane < 6) || lane >= 12) lev = (lev + R) - R;
    const double sa = __shfl_sync(0xffffffffu, lev, lane == 8 ? 13 : 12), sb = __shfl_sync(0xffffffffu, lev, lane == 6 ? 13 : 14);
    const double a = __shfl_sync(0xffffffffu, lev, (lane - 3) & 31);
    if (lane >= 6 && lane < 9) lev = (sa + sb) - a;
  }
  if (lane < 15) M.lev[lane] = lev * (lane < 3 ? 0.25 : lane < 9 ? 1.0 : lane < 12 ? 0.5 : 2.0);
}

// The six covariance entries of one bin or layer from the model's sums and the
// transfer products (table rows kTabU1 .. kTabV2).
__device__ __forceinline__ void noise_inst_cov(const NoiseModel &M, double u1, double u2, double u3, double v1,
                                               double v2, double *c) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    c[k] = fma(u1, M.lev[k], fma(u2, M.lev[3 + k], u3 * M.lev[6 + k]));
    c[3 + k] = fma(v1, M.lev[9 + k], v2 * M.lev[12 + k]);
  }
}

// exp(2 (f - fk) / f2), for the foreground's 0.5 (1 + tanh((fk - f) / f2)) =
// 1 / (1 + E).
__device__ __forceinline__ double noise_gal_exp(const NoiseModel &M, double f, const double *t) {
  return exp_tab((f - M.fk) * M.i2, t);
}
// The galactic foreground's PSD at f (utils/src/glass_galaxy.c:40-44), zero
// above 10 f1 as in noise/src/glass_noise_model.c:627-631; fp73 = f^(-7/3),
// lf = log f, E as above.
__device__ __forceinline__ double noise_sgal(const NoiseModel &M, double f, double fp73, double lf, double E,
                                             const double *t) {
  if (f > M.f10) return 0.0;
  const double u = exp_tab(M.alpha * (lf - M.l1), t);
  const int h = __double2hiint(E);
  const double w = (h >= 0x7e000000 && h <= 0x7ff00000) ? 0.0 : rcp_fast(1.0 + E);  // E beyond 2^993: tanh = -1
  return M.Amp * fp73 * exp_tab(-u, t) * w;
}

// ------------------------------------------------------------------ SGWB
// Cosmological constants of the templates (utils/src/glass_constants.h:81-86):
// H0 = 70 km/s/Mpc in 1/s, the f^-3 prefactor 3 H0^2 / (4 pi^2) that turns
// an energy-density spectrum into a strain PSD, and the radiation-era
// transfer factor of the lognormal template.
constexpr double kSgH0 = 70 * 3.24078e-20;
constexpr double kSgHscale = 3 * kSgH0 * kSgH0 / (4 * M_PI * M_PI);
constexpr double kSgCgOr0 = 1.6e-5 / (0.7 * 0.7);

// erfc by Abramowitz & Stegun 7.1.26 (|error| < 1.5e-7), the rational
// approximation the reference's glass_erfc uses (utils/src/glass_math.c:1310),
// evaluated on |x| and reflected (erfc(-x) = 2 - erfc(x)).
__device__ __forceinline__ double sgwb_erfc(double x) {
  const double ax = fabs(x);
  const double t = 1.0 / (1.0 + 0.3275911 * ax);
  const double poly = ((((1.061405429 * t - 1.453152027) * t + 1.421413741) * t - 0.284496736) * t + 0.254829592) * t;
  const double y = poly * exp(-ax * ax);
  return x < 0.0 ? 2.0 - y : y;
}

// The background's strain PSD at f > 0 (noise/src/glass_noise_model.c:725-776):
//  powerlaw          p = log10 A, alpha: A (f / 25 Hz)^alpha
//  lognormal         p = log10 A, log10 f*, log10 Delta: the wide-Delta
//                    lognormal-peak spectrum of Pi & Sasaki (JCAP 2020,
//                    eq. 3.29), its asymptote 0.783e-3 A^2 for Delta >= 9
//  phase transition  p = rb, b, log10 Ap, log10 fp: Ap times the broken power
//                    law in s = f / fp with slopes 9 and b
// each times Hscale / f^3.
__device__ double sgwb_psd(int type, double f, const double *p) {
  const double pre = kSgHscale / (f * f * f);
  if (type == kSgwbPowerlaw) {
    const double A = pow(10.0, p[0]);
    return pre * A * pow(f / 25.0, p[1]);
  }
  if (type == kSgwbLognormal) {
    const double A = pow(10.0, p[0]), fst = pow(10.0, p[1]), D = pow(10.0, p[2]);
    const double scale = pre * kSgCgOr0 * A * A;
    if (!(D < 9.0)) return scale * 0.783 / 1e3;
    const double ft = f / fst, lft = log(ft), D2 = D * D;
    const double rpi = sqrt(M_PI);
    const double h32 = 0.5 * log(1.5);
    const double lK = lft + 1.5 * D2;
    const double u = lK + h32;
    const double t1 = 4.0 / 5.0 / rpi * ft * ft * ft * exp(9.0 * D2 / 4.0) / D *
                      ((lK * lK + 0.5 * D2) * sgwb_erfc(u / D) - D / rpi * exp(-u * u / D2) * (lK - h32));
    const double v = lft + D2 - 0.5 * log(4.0 / 3.0);
    const double t2 = 0.0659 / D2 * ft * ft * exp(D2) * exp(-v * v / D2);
    const double t3 = (1.0 / 3.0) * sqrt(2.0) / rpi * pow(ft, -4) * exp(8.0 * D2) / D * exp(-lft * lft / (2.0 * D2)) *
                      sgwb_erfc((4.0 * D2 - lft + log(4.0)) / (D * sqrt(2.0)));
    return scale * (t1 + t2 + t3);
  }
  // phase transition
  const double rb = p[0], b = p[1], Ap = pow(10.0, p[2]), fp = pow(10.0, p[3]);
  const double rb4 = rb * rb * rb * rb;
  const double m = (9 * rb4 + b) / (rb4 + 1);
  const double sr = f / fp, s4 = sr * sr * sr * sr, s9 = s4 * s4 * sr;
  const double M = s9 * pow((1 + rb4) / (rb4 + s4), (9 - b) / 4) * pow((b + 4) / (b + 4 - m + m * sr * sr), (b + 4) / 2);
  return Ap * M * pre;
}

// Inverse and log-determinant of a symmetric 3x3 covariance by the
// reference's elimination (utils/src/glass_math.c:261-274), the entries as
// cofactor / det: iv = xx, yy, zz, xy, xz, yz.
__device__ __forceinline__ void noise_inv3(double cxx, double cyy, double czz, double cxy, double cxz, double cyz,
                                           double *iv, double &logdetC) {
  const double d1 = cxx;
  const double d2 = cyy - cxy * cxy / d1;
  const double tt = cyz - cxy * cxz / d1;
  const double d3 = (czz - cxz * cxz / d1) - (tt * tt) / d2;
  logdetC = log(d1) + log(d2) + log(d3);
  const double idet = 1.0 / (d1 * d2 * d3);
  iv[0] = (cyy * czz - cyz * cyz) * idet;
  iv[1] = (czz * cxx - cxz * cxz) * idet;
  iv[2] = (cxx * cyy - cxy * cxy) * idet;
  iv[3] = (cxz * cyz - czz * cxy) * idet;
  iv[4] = (cxy * cyz - cxz * cyy) * idet;
  iv[5] = (cxy * cxz - cxx * cyz) * idet;
}

// chi^2 + log det of one cell by the elimination above, for covariances the
// fast form does not take (not positive, not finite, or with a determinant at
// the ends of the exponent range).
__device__ __noinline__ double noise_cell_general(double cxx, double cyy, double czz, double cxy, double cxz,
                                                  double cyz, const double *P) {
  double iv[6], ld;
  noise_inv3(cxx, cyy, czz, cxy, cxz, cyz, iv, ld);
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 6; k++) s += P[k] * iv[k];
  return s + ld;
}

// Adds tr(C^-1 P) and log det C of one cell, c = xx, yy, zz, xy, xz, yz and
// P = xx, yy, zz, 2 xy, 2 xz, 2 yz: 12 operations for the cofactors, 3 for the
// determinant, 6 for the trace's numerator, 3 for the reciprocal, 2 for the sums.
// The determinant's cancellation where the channels are nearly degenerate
// (third pivot ~1e-7 of the first at 0.1 mHz) is that of the elimination's.
__device__ __forceinline__ void noise_cell(const double *c, const double *P, double &chi, LogSum &ld) {
  const double cxx = c[0], cyy = c[1], czz = c[2], cxy = c[3], cxz = c[4], cyz = c[5];
  const double m2 = fma(cxx, cyy, -(cxy * cxy));
  const double m4 = fma(cxy, cyz, -(cxz * cyy));
  const double m5 = fma(cxy, cxz, -(cxx * cyz));
  const double det = fma(czz, m2, fma(cyz, m5, cxz * m4));
  // all leading minors positive, as the reference's logarithms need
  if (__double2hiint(cxx) > 0 && __double2hiint(m2) > 0 && plain_positive(det)) {
    const double m0 = fma(cyy, czz, -(cyz * cyz));
    const double m1 = fma(czz, cxx, -(cxz * cxz));
    const double m3 = fma(cxz, cyz, -(czz * cxy));
    double num = m0 * P[0];
    num = fma(m1, P[1], num);
    num = fma(m2, P[2], num);
    num = fma(m3, P[3], num);
    num = fma(m4, P[4], num);
    num = fma(m5, P[5], num);
    chi = fma(num, rcp_fast(det), chi);
    log_add(ld, det);
  } else {
    chi += noise_cell_general(cxx, cyy, czz, cxy, cxz, cyz, P);
  }
}

// One CTA per (chunk of 128 R bins, model): per-bin covariance, inverse and
// likelihood terms; the chunk's sum goes to partial[model][chunk].  Bound by
// the FP64 pipe (see the top of the file).
__global__ void __launch_bounds__(kNoiseThreads) noise_logl_kernel(NoiseArgs a) {
  grid_begin();
  __shared__ double et[kExpTab];
  __shared__ NoiseModel M;
  const int chunk = blockIdx.x, p = blockIdx.y;
  const bool gal = a.sgal != nullptr;
  noise_model_load(M, a.inst + 12 * (size_t)p, gal ? a.sgal + 5 * (size_t)p : nullptr, a.fstep);
  if (gal) exp_tab_fill(et);
  __syncthreads();
  const double *sgp = a.sgwb ? a.sgwb + 4 * (size_t)p : nullptr;
  const size_t N = a.N;
  double chi = 0.0, E = 0.0;
  LogSum ld;
#pragma unroll 1
  for (int r = 0; r < a.R; r++) {
    const int n = (chunk * a.R + r) * kNoiseThreads + threadIdx.x;
    if (n >= a.N) break;
    const double *t = a.tab + n;
    double c[6], P[6];
    noise_inst_cov(M, t[kTabU1 * N], t[kTabU2 * N], t[kTabU3 * N], t[kTabV1 * N], t[kTabV2 * N], c);
    if (gal) {
      const double f = t[kTabF * N];
      E = (r > 0 && M.chain) ? E * M.estep : noise_gal_exp(M, f, et);
      const double S = noise_sgal(M, f, t[kTabFp73 * N], t[kTabLogf * N], E, et);
      const double d = 0.25 * t[kTabTgal * N] * S;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        c[k] += d;
        c[3 + k] = fma(-0.5, d, c[3 + k]);
      }
    }
    if (sgp) {
      // added last, as the instrument sampler combines the three
      // (noise/src/glass_noise_sampler.c:559-568)
      const double f = t[kTabF * N];
      const double S = f != 0.0 ? sgwb_psd(a.sg_type, f, sgp) : 0.0;
#pragma unroll
      for (int k = 0; k < 6; k++) c[k] = fma(a.rsg[k * N + n], S, c[k]);
    }
#pragma unroll
    for (int k = 0; k < 6; k++) P[k] = t[(kTabXX + k) * N];
    noise_cell(c, P, chi, ld);
  }
  const double s = block_total(chi, ld);
  if (threadIdx.x == 0) a.partial[(size_t)p * a.nchunks + chunk] = -s;
}

// The one- and two-channel forms: the instrument covariance of
// generate_instrument_noise_model's case 1 (Michelson X, XYZnoise_FF) and
// case 2 (A and E, AEnoise_FF; utils/src/glass_lisa.c:1121-1145) on the link
// levels sacc12 = in[0], soms12 = in[6] (noise/src/glass_noise_model.c:450-461),
// normalised by 4, plus the foreground's case 1 (Sgal / 4) or case 2
// (1.5 t Sgal / 4, :635-641), the diagonal inverse and log-determinant
// (utils/src/glass_math.c:248-258) and noise_log_likelihood's sum
// (noise/src/glass_noise_model.c:1104-1134).  sin^2(f/f*) is the table's
// -8 sin^2 times -1/8 (exact).
__global__ void __launch_bounds__(kNoiseThreads) noise_ch12_kernel(NoiseArgs a, int nch) {
  grid_begin();
  __shared__ double et[kExpTab];
  __shared__ NoiseModel M;
  const int chunk = blockIdx.x, p = blockIdx.y;
  const double *in = a.inst + 12 * (size_t)p;
  const bool gal = a.sgal != nullptr;
  noise_model_load(M, in, gal ? a.sgal + 5 * (size_t)p : nullptr, a.fstep);
  if (gal) exp_tab_fill(et);
  __syncthreads();
  const double sacc12 = in[0], soms12 = in[6];
  const size_t N = a.N;
  double chi = 0.0, E = 0.0;
  LogSum ld;
#pragma unroll 1
  for (int r = 0; r < a.R; r++) {
    const int n = (chunk * a.R + r) * kNoiseThreads + threadIdx.x;
    if (n >= a.N) break;
    const double *t = a.tab + n;
    const double f = t[kTabF * N];
    double c = 0.0;
    if (f != 0.0) {
      const double cosx = t[kTabCosx * N], sx2 = t[kTabTdi * N] * -0.125;
      const double Spm = sacc12 * t[kTabAcc * N], Sop = soms12 * t[kTabOms * N];
      c = (nch == 1) ? 16. * sx2 * (2. * (1.0 + cosx * cosx) * Spm + Sop)
                     : 8. * sx2 * (2. * Spm * (3. + 2. * cosx + t[kTabCos2x * N]) + Sop * (2. + cosx));
      c = c * 0.25;
      if (gal) {
        E = (r > 0 && M.chain) ? E * M.estep : noise_gal_exp(M, f, et);
        const double Sgal = noise_sgal(M, f, t[kTabFp73 * N], t[kTabLogf * N], E, et);
        c += (nch == 1 ? Sgal : 1.5 * t[kTabTgal * N] * Sgal) * 0.25;
      }
    }
    const double P = nch == 2 ? t[kTabP0 * N] + t[kTabP1 * N] : t[kTabP0 * N];
    if (plain_positive(c)) {
      chi = fma(P, rcp_fast(c), chi);
      log_add(ld, c);
      if (nch == 2) log_add(ld, c);
    } else {
      chi += P * (1. / c) + (nch == 2 ? 2.0 : 1.0) * log(c);
    }
  }
  const double s = block_total(chi, ld);
  if (threadIdx.x == 0) a.partial[(size_t)p * a.nchunks + chunk] = -s;
}

// Per model: the chunks' sums in order, and the constant -3 N log(2 pi).
__global__ void noise_finish_kernel(const double *partial, int nchunks, int nprop, double cst, double *logl) {
  grid_begin();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nprop) return;
  double s = 0.0;
  for (int c = 0; c < nchunks; c++) s += partial[(size_t)p * nchunks + c];
  logl[p] = s - cst;
}


// ------------------------------------------------------- wavelet domain
struct NoiseWvArgs {
  int Nlayer, Ncoarse, Q, LJ, nchunks, mode;
  double inv_ND;
  const double *tab, *P, *mod;
  const double *inst, *sgal;
  int sg_type;
  const double *sgwb, *rsg;  // [nprop][4] or null; 6 rows of Nlayer
  double *out;  // logl (modes 0/1) or partial (mode 2)
};

// One layer's covariances in the wavelet domain: the Fourier model at the layer
// centre over ND (generate_instrument_noise_model_wavelet :561-610), plus the
// background's (generate_sgwb_model_wavelet :843-892, zero in the DC layer), in
// c6 = xx, yy, zz, xy, xz, yz; returns the foreground's (generate_galactic_
// foreground_model_wavelet :656-722), the same for the three diagonal and, with
// the isotropic -1/2 undone, for the three off-diagonal entries.
__device__ __forceinline__ double noise_wv_layer(const NoiseWvArgs &a, const NoiseModel &M, int j, bool gal,
                                                 const double *sgp, const double *et, double *c6) {
  const size_t NL = a.Nlayer;
  const double *t = a.tab + j;
  const double f = t[kTabF * NL];
  noise_inst_cov(M, t[kTabU1 * NL], t[kTabU2 * NL], t[kTabU3 * NL], t[kTabV1 * NL], t[kTabV2 * NL], c6);
#pragma unroll
  for (int e = 0; e < 6; e++) c6[e] *= a.inv_ND;
  if (sgp && f != 0.0) {
    const double S = sgwb_psd(a.sg_type, f, sgp) * a.inv_ND;
#pragma unroll
    for (int e = 0; e < 6; e++) c6[e] = fma(a.rsg[e * NL + j], S, c6[e]);
  }
  if (!gal || f == 0.0) return 0.0;
  const double S = noise_sgal(M, f, t[kTabFp73 * NL], t[kTabLogf * NL], noise_gal_exp(M, f, et), et);
  return 0.25 * t[kTabTgal * NL] * S * a.inv_ND;
}

// Modes 0/1: the covariance is the same for every cell of a layer, so a
// layer's cells contribute -Q/2 (ixx Sxx + ... + 2 ixy Sxy ...) - Q/2 Ncoarse
// log det with S the layer's sums of the cell statistics.  One CTA per model.
__global__ void __launch_bounds__(kNoiseThreads) noise_wv_stationary_kernel(NoiseWvArgs a) {
  grid_begin();
  __shared__ double et[kExpTab];
  __shared__ NoiseModel M;
  const int p = blockIdx.x;
  const bool gal = a.mode == 1;
  noise_model_load(M, a.inst + 12 * (size_t)p, gal ? a.sgal + 5 * (size_t)p : nullptr, 0.0);
  if (gal) exp_tab_fill(et);
  __syncthreads();
  const size_t NL = a.Nlayer;
  const double *sgp = a.sgwb ? a.sgwb + 4 * (size_t)p : nullptr;
  const double cells = (double)a.Ncoarse, icells = 1.0 / cells;
  double chi = 0.0;
  LogSum ld;
  for (int j = threadIdx.x; j < a.Nlayer; j += blockDim.x) {
    double c6[6], P[6];
    // generate_full_stationary_covariance_matrix_coarse (:1003-1010)
    const double g = noise_wv_layer(a, M, j, gal, sgp, et, c6);
#pragma unroll
    for (int e = 0; e < 3; e++) {
      c6[e] += g;
      c6[3 + e] = fma(-0.5, g, c6[3 + e]);
      P[e] = a.tab[(kTabXX + e) * NL + j] * icells;
      P[3 + e] = a.tab[(kTabXY + e) * NL + j] * icells;
    }
    noise_cell(c6, P, chi, ld);
  }
  const double s = block_total(chi, ld);
  if (threadIdx.x == 0) a.out[p] = -0.5 * (double)a.Q * cells * s;
}

// Mode 2: the foreground modulated per cell (generate_full_dynamic_covariance_
// matrix_coarse :923-981).  One CTA per (chunk of LJ layers, model); the
// chunk's layer covariances go to shared memory, then every cell is inverted
// and summed with its statistics (my_noise_log_likelihood_wavelet_coarse
// :1211-1241): 6 FP64 operations for its covariance, 26 in noise_cell.
constexpr int kNoiseWvMaxLJ = 64;
__global__ void __launch_bounds__(kNoiseThreads) noise_wv_dynamic_kernel(NoiseWvArgs a) {
  grid_begin();
  __shared__ double et[kExpTab];
  __shared__ double lay[kNoiseWvMaxLJ][7];
  __shared__ NoiseModel M;
  const int chunk = blockIdx.x, p = blockIdx.y;
  noise_model_load(M, a.inst + 12 * (size_t)p, a.sgal + 5 * (size_t)p, 0.0);
  exp_tab_fill(et);
  __syncthreads();
  const double *sgp = a.sgwb ? a.sgwb + 4 * (size_t)p : nullptr;
  const int j0 = chunk * a.LJ;
  const int nl = min(a.LJ, a.Nlayer - j0);
  if ((int)threadIdx.x < nl) {
    double c6[6];
    lay[threadIdx.x][6] = noise_wv_layer(a, M, j0 + threadIdx.x, true, sgp, et, c6);
#pragma unroll
    for (int e = 0; e < 6; e++) lay[threadIdx.x][e] = c6[e];
  }
  __syncthreads();
  const int Nc = a.Ncoarse;
  const size_t Npix = (size_t)a.Nlayer * Nc;
  double chi = 0.0;
  LogSum ld;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < nl * Nc; idx += blockDim.x) {
    const int jj = idx / Nc, q = idx - jj * Nc;
    const double *P0 = a.P + (size_t)j0 * Nc + idx;
    double c6[6], P[6];
#pragma unroll
    for (int e = 0; e < 6; e++) {
      c6[e] = fma(lay[jj][6], a.mod[(size_t)e * Nc + q], lay[jj][e]);
      P[e] = P0[e * Npix];
    }
    noise_cell(c6, P, chi, ld);
  }
  const double s = block_total(chi, ld);
  if (threadIdx.x == 0) a.out[(size_t)p * a.nchunks + chunk] = -0.5 * (double)a.Q * s;
}

__global__ void noise_wv_const_kernel(double *logl, int nprop, double cst) {
  grid_begin();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < nprop) logl[p] -= cst;
}

// ------------------------------------------------ spline noise model
// One CTA per model (noise_spline_model_mcmc / _rjmcmc,
// noise/src/glass_noise_sampler.c:133, :232): one thread per channel solves
// the natural cubic spline through the model's control points
// (spline_coefficients, utils/src/glass_math.c:98-178: the tridiagonal
// system's forward elimination and back substitution, sequential), then all
// threads evaluate it over the bins with the binary-search lookup (the largest
// knot <= f: binary_search, :443-473, on distinct knots), add the transfer
// floor (generate_spline_noise_model, noise/src/glass_noise_model.c:366-387),
// and sum noise_log_likelihood's terms (:1104-1134): -|d|^2 / C per channel
// and -log C.
struct SplineNoiseArgs {
  int nch, N, kmax;
  const double *tab;  // f, transfer, P0[, P1]
  const int *nknots;
  const double *knot_f, *knot_C;
  double *logl;
};

__device__ __forceinline__ int spline_knot_below(int K, const double *x, double v) {
  if (v <= x[0]) return 0;
  if (v >= x[K - 1]) return K - 1;
  int lo = 0, hi = K - 1;  // x[lo] <= v < x[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (x[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

constexpr int kSplineThreads = 256;

__device__ __forceinline__ double block_sum(double v, double *red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kSplineThreads / 32; w++) s += red[w];
  return s;
}

__global__ void __launch_bounds__(kSplineThreads) spline_noise_kernel(SplineNoiseArgs a) {
  extern __shared__ double sm[];
  __shared__ double red[kSplineThreads / 32];
  const int p = blockIdx.x, K = a.nknots[p], KM = a.kmax;
  if (K < 2 || K > KM) {  // the whole CTA leaves before any barrier
    if (threadIdx.x == 0) a.logl[p] = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
  // x[KM], then per channel c0, c1, c2, c3, mu, z (each KM)
  double *x = sm;
  for (int k = threadIdx.x; k < K; k += blockDim.x) x[k] = a.knot_f[(size_t)p * KM + k];
  __syncthreads();
  if (threadIdx.x < a.nch) {
    const int c = threadIdx.x;
    double *c0 = sm + KM * (1 + 6 * c), *c1 = c0 + KM, *c2 = c1 + KM, *c3 = c2 + KM, *mu = c3 + KM, *z = mu + KM;
    const double *y = a.knot_C + ((size_t)p * a.nch + c) * KM;
    mu[0] = z[0] = 0.0;
    for (int i = 1; i < K - 1; i++) {
      const double hm = x[i] - x[i - 1], hi = x[i + 1] - x[i];
      const double al = 3.0 * ((y[i + 1] - y[i]) / hi - (y[i] - y[i - 1]) / hm);
      const double l = 2.0 * (x[i + 1] - x[i - 1]) - hm * mu[i - 1];
      mu[i] = hi / l;
      z[i] = (al - hm * z[i - 1]) / l;
    }
    c0[K - 1] = y[K - 1];
    c1[K - 1] = c2[K - 1] = c3[K - 1] = 0.0;
    for (int i = K - 2; i >= 0; i--) {
      const double h = x[i + 1] - x[i];
      c0[i] = y[i];
      c2[i] = z[i] - mu[i] * c2[i + 1];
      c1[i] = (c0[i + 1] - c0[i]) / h - h * (c2[i + 1] + 2.0 * c2[i]) / 3.0;
      c3[i] = (c2[i + 1] - c2[i]) / (3.0 * h);
    }
  }
  __syncthreads();
  const int N = a.N;
  const double *F = a.tab, *TR = a.tab + N;
  double acc = 0.0;
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    const double f = F[n];
    const int j = spline_knot_below(K, x, f);
    const double d = f - x[j];
    double ld = 0.0;
    for (int c = 0; c < a.nch; c++) {
      const double *c0 = sm + KM * (1 + 6 * c), *c1 = c0 + KM, *c2 = c1 + KM, *c3 = c2 + KM;
      const double C = (c0[j] + c1[j] * d + c2[j] * d * d + c3[j] * d * d * d) + TR[n];
      acc -= 0.5 * (2.0 * (a.tab[(size_t)(2 + c) * N + n] * (1. / C)));
      ld += log(C);
    }
    acc -= ld;
  }
  const double s = block_sum(acc, red);
  if (threadIdx.x == 0) a.logl[p] = s;
}

}  // namespace

// ------------------------------------------------------------------- host
// The per-bin table, with the reference's own expressions (host libm): the
// grid f_n = fmin + n/T (noise/src/glass_noise_model.c:1384-1385), the
// transfer functions of :415-446 and :620-624, and the data's auto- and
// cross-spectra of :1251-1263.
static void noise_freq_rows(double f, double *tab, int N, int n) {
  const double fstar = kCLIGHT / (2.0 * M_PI * kLARM);
  const double acc_units = 2.81837551648e-19;  // 1/(2 pi c)^2
  const double oms_units = 4.39256635604e-16;  // (2 pi / c)^2
  const double acc_fmax = 0.01;
  double *col[kNoiseTabRows];
  for (int r = 0; r < kNoiseTabRows; r++) col[r] = tab + (size_t)r * N + n;
  *col[kTabF] = f;
  if (f != 0.0) {
    const double x = f / fstar, f2 = f * f;
    const double sx = sin(x);
    *col[kTabCosx] = cos(x);
    *col[kTabTdi] = -8.0 * (sx * sx);
    *col[kTabAcc] = (f < acc_fmax) ? acc_units / f2 * (1.0 + pow(0.4e-3 / f, 2)) * (1.0 + pow(f / 8.0e-3, 4)) : 0.0;
    *col[kTabOms] = oms_units * f2 * (1.0 + pow(2.0e-3 / f, 4));
    const double xg = f / (kCLIGHT / (kPI2 * kLARM));
    *col[kTabTgal] = 4. * xg * xg * sin(xg) * sin(xg);
    *col[kTabFp73] = pow(f, -7. / 3.);
    *col[kTabLogf] = log(f);
  } else {
    *col[kTabCosx] = *col[kTabTdi] = *col[kTabAcc] = *col[kTabOms] = *col[kTabTgal] = *col[kTabFp73] = 0.0;
    *col[kTabLogf] = 0.0;
  }
  // the covariance's products (the reference's c_ij / 4)
  const double cx = *col[kTabCosx], td = *col[kTabTdi];
  *col[kTabU1] = -0.5 * td * *col[kTabOms];
  *col[kTabU2] = -0.5 * td * *col[kTabAcc];
  *col[kTabU3] = *col[kTabU2] * cx * cx;
  *col[kTabV1] = 0.25 * td * cx * *col[kTabOms];
  *col[kTabV2] = 0.25 * td * cx * *col[kTabAcc];
}

void noise_build_table(double T, double fmin, int N, const double *X, const double *Y, const double *Z,
                       double *tab) {
  for (int n = 0; n < N; n++) {
    noise_freq_rows(fmin + (double)n / T, tab, N, n);
    const double rex = X[2 * n], imx = X[2 * n + 1];
    const double rey = Y[2 * n], imy = Y[2 * n + 1];
    const double rez = Z[2 * n], imz = Z[2 * n + 1];
    tab[(size_t)kTabXX * N + n] = rex * rex + imx * imx;
    tab[(size_t)kTabYY * N + n] = rey * rey + imy * imy;
    tab[(size_t)kTabZZ * N + n] = rez * rez + imz * imz;
    tab[(size_t)kTabXY * N + n] = 2.0 * (rex * rey + imx * imy);
    tab[(size_t)kTabXZ * N + n] = 2.0 * (rex * rez + imx * imz);
    tab[(size_t)kTabYZ * N + n] = 2.0 * (rey * rez + imy * imz);
  }
}

void noise_build_table_ch(double T, double fmin, int N, int nch, const double *d0, const double *d1, double *tab) {
  const double fstar = kCLIGHT / (2.0 * M_PI * kLARM);
  for (int n = 0; n < N; n++) {
    const double f = fmin + (double)n / T;
    noise_freq_rows(f, tab, N, n);
    tab[(size_t)kTabCos2x * N + n] = cos(2. * (f / fstar));  // AEnoise_FF's cos 2x
    tab[(size_t)kTabP0 * N + n] = d0[2 * n] * d0[2 * n] + d0[2 * n + 1] * d0[2 * n + 1];
    tab[(size_t)kTabP1 * N + n] = nch == 2 ? d1[2 * n] * d1[2 * n] + d1[2 * n + 1] * d1[2 * n + 1] : 0.0;
    for (int r = kTabXY; r <= kTabYZ; r++) tab[(size_t)r * N + n] = 0.0;
  }
}

void noise_wv_build(int NT, double df, int lmin, int Nlayer, int Q, const double *X, const double *Y, const double *Z,
                    double *tab, double *P) {
  const int Nc = NT / Q;
  const size_t Npix = (size_t)Nlayer * Nc;
  const double invQ = 1.0 / (double)Q;
  for (int j = 0; j < Nlayer; j++) {
    noise_freq_rows((double)(lmin + j) * df, tab, Nlayer, j);
    double S[6] = {0, 0, 0, 0, 0, 0};
    for (int q = 0; q < Nc; q++) {
      double sxx = 0, syy = 0, szz = 0, sxy = 0, sxz = 0, syz = 0;
      for (int i = q * Q; i < (q + 1) * Q; i++) {
        const size_t k = (size_t)i + (size_t)j * NT;
        const double wx = X[k], wy = Y[k], wz = Z[k];
        sxx += wx * wx;
        syy += wy * wy;
        szz += wz * wz;
        sxy += wx * wy;
        sxz += wx * wz;
        syz += wy * wz;
      }
      const size_t kc = (size_t)q + (size_t)j * Nc;
      const double v[6] = {sxx * invQ, syy * invQ, szz * invQ, 2.0 * (sxy * invQ), 2.0 * (sxz * invQ),
                           2.0 * (syz * invQ)};  // the off-diagonal terms count twice
      for (int e = 0; e < 6; e++) {
        P[(size_t)e * Npix + kc] = v[e];
        S[e] += v[e];
      }
    }
    for (int e = 0; e < 6; e++) tab[(size_t)(kTabXX + e) * Nlayer + j] = S[e];
  }
}

// Natural cubic spline through (x[i], y[i]) in the coefficient form
// y0 + y1 d + y2 d^2 + y3 d^3 on interval i (the tridiagonal solve of
// spline_coefficients, utils/src/glass_math.c:98-178), evaluated with the
// even-spacing lookup of even_sampled_search (:393-402: floor of the offset
// over x[1] - x[0], clamped to [0, n - 1]; the last node's polynomial is the
// constant y[n - 1]).
namespace {
struct SgSpline {
  std::vector<double> x, c0, c1, c2, c3;
  void fit(const std::vector<double> &xs, const std::vector<double> &ys) {
    const int n = (int)xs.size();
    x = xs;
    c0.assign(n, 0.0);
    c1.assign(n, 0.0);
    c2.assign(n, 0.0);
    c3.assign(n, 0.0);
    std::vector<double> h(n, 0.0), rhs(n, 0.0), diag(n, 1.0), up(n, 0.0), z(n, 0.0);
    h[0] = xs[1] - xs[0];
    for (int i = 1; i < n - 1; i++) {
      h[i] = xs[i + 1] - xs[i];
      rhs[i] = 3.0 * ((ys[i + 1] - ys[i]) / h[i] - (ys[i] - ys[i - 1]) / h[i - 1]);
    }
    for (int i = 1; i < n - 1; i++) {  // forward elimination, natural ends
      diag[i] = 2.0 * (xs[i + 1] - xs[i - 1]) - h[i - 1] * up[i - 1];
      up[i] = h[i] / diag[i];
      z[i] = (rhs[i] - h[i - 1] * z[i - 1]) / diag[i];
    }
    c0[n - 1] = ys[n - 1];
    for (int i = n - 2; i >= 0; i--) {  // back substitution
      c0[i] = ys[i];
      c2[i] = z[i] - up[i] * c2[i + 1];
      c1[i] = (c0[i + 1] - c0[i]) / h[i] - h[i] * (c2[i + 1] + 2.0 * c2[i]) / 3.0;
      c3[i] = (c2[i + 1] - c2[i]) / (3.0 * h[i]);
    }
  }
  double at(double v) const {
    const int n = (int)x.size();
    int j = (int)floor((v - x[0]) / (x[1] - x[0]));
    if (j < 0) j = 0;
    if (j > n - 1) j = n - 1;
    const double d = v - x[j];
    return c0[j] + c1[j] * d + c2[j] * d * d + c3[j] * d * d * d;
  }
};
}  // namespace

int noise_sgwb_rows(int nresp, const double *resp, int N, const double *f, double *R6) {
  // alloc_pop_sgwb_response (noise/src/glass_noise_model.c:134-189): 10 to
  // 3000 rows; log of f and of the auto-responses, asinh of the
  // cross-responses over 1e-7
  if (nresp < 10 || nresp > 3000) return -1;
  const double ascale = 1e-7;
  std::vector<double> lf(nresp), col[6];
  for (int e = 0; e < 6; e++) col[e].resize(nresp);
  for (int i = 0; i < nresp; i++) {
    const double *r = resp + 7 * (size_t)i;
    if (!(r[0] > 0) || !(r[1] > 0) || !(r[2] > 0) || !(r[3] > 0)) return -1;
    lf[i] = log(r[0]);
    for (int e = 0; e < 3; e++) col[e][i] = log(r[1 + e]);
    for (int e = 3; e < 6; e++) col[e][i] = asinh(r[1 + e] / ascale);
  }
  SgSpline sp[6];
  for (int e = 0; e < 6; e++) sp[e].fit(lf, col[e]);
  for (int n = 0; n < N; n++) {
    if (f[n] == 0.0) {
      for (int e = 0; e < 6; e++) R6[(size_t)e * N + n] = 0.0;
      continue;
    }
    const double l = log(f[n]);  // generate_sgwb_model (:808-820)
    for (int e = 0; e < 3; e++) R6[(size_t)e * N + n] = exp(sp[e].at(l));
    for (int e = 3; e < 6; e++) R6[(size_t)e * N + n] = ascale * sinh(sp[e].at(l));
  }
  return 0;
}

// Layers per CTA of the modulated form: about 4096 cells, fewer where the
// batch is too small to give every SM a few CTAs (a CTA's model constants and
// layer covariances cost about as much as 300 cells).
int noise_wv_layers_per_cta(int Nlayer, int Ncoarse, int nprop, int num_sms) {
  int lj = 4096 / (Ncoarse > 0 ? Ncoarse : 1);
  if (lj < 1) lj = 1;
  if (lj > kNoiseWvMaxLJ) lj = kNoiseWvMaxLJ;
  while (lj > 1 && (long long)((Nlayer + lj - 1) / lj) * nprop < (long long)kNoiseCtasPerSm * num_sms) lj = (lj + 1) / 2;
  return lj;
}

// As noise_partials.
size_t noise_wv_partials(int Nlayer, int Ncoarse, int nprop, int num_sms) {
  const int lj = noise_wv_layers_per_cta(Nlayer, Ncoarse, 1 << 30, num_sms);
  const size_t most = (size_t)nprop * ((Nlayer + lj - 1) / lj);
  const size_t few = 2 * (size_t)kNoiseCtasPerSm * num_sms + 2 * (size_t)nprop;
  return most > few ? most : few;
}

cudaError_t noise_wv_logl_launch(const NoiseWvDev &w, int mode, int nprop, const double *inst, const double *sgal,
                                 int sg_type, const double *sgwb, double *logl, int num_sms, cudaStream_t stream,
                                 int *nlaunch) {
  NoiseWvArgs a;
  a.Nlayer = w.Nlayer;
  a.Ncoarse = w.Ncoarse;
  a.Q = w.Q;
  a.LJ = noise_wv_layers_per_cta(w.Nlayer, w.Ncoarse, nprop, num_sms);
  a.nchunks = (w.Nlayer + a.LJ - 1) / a.LJ;
  a.mode = mode;
  a.inv_ND = 1.0 / (double)((long long)w.NF * w.NT);
  a.tab = w.tab;
  a.P = w.P;
  a.mod = w.mod;
  a.inst = inst;
  a.sgal = sgal;
  a.sg_type = sg_type;
  a.sgwb = sgwb;
  a.rsg = w.rsg;
  int launches = 0;
  cudaError_t e;
  if (mode != 2) {
    for (int p0 = 0; p0 < nprop; p0 += 65535 * 16) {
      const int np = nprop - p0 < 65535 * 16 ? nprop - p0 : 65535 * 16;
      NoiseWvArgs s = a;
      s.inst = inst + 12 * (size_t)p0;
      s.sgal = sgal ? sgal + 5 * (size_t)p0 : nullptr;
      s.sgwb = sgwb ? sgwb + 4 * (size_t)p0 : nullptr;
      s.out = logl + p0;
      launches++;
      if ((e = launch_chained(noise_wv_stationary_kernel, np, kNoiseThreads, 0, stream, s)) != cudaSuccess) return e;
    }
  } else {
    for (int p0 = 0; p0 < nprop; p0 += 65535) {
      const int np = nprop - p0 < 65535 ? nprop - p0 : 65535;
      NoiseWvArgs s = a;
      s.inst = inst + 12 * (size_t)p0;
      s.sgal = sgal + 5 * (size_t)p0;
      s.sgwb = sgwb ? sgwb + 4 * (size_t)p0 : nullptr;
      s.out = w.partial + (size_t)p0 * a.nchunks;
      launches++;
      if ((e = launch_chained(noise_wv_dynamic_kernel, dim3(a.nchunks, np), kNoiseThreads, 0, stream, s)) != cudaSuccess)
        return e;
    }
  }
  // my_noise_log_likelihood_wavelet_coarse's constant over the full pixel count (:1238-1240)
  const double cst = 0.5 * 3 * ((double)w.Nlayer * w.NT) * log(2 * M_PI);
  launches++;
  if (nlaunch) *nlaunch = launches;
  if (mode == 2)
    return launch_chained(noise_finish_kernel, (nprop + 255) / 256, 256, 0, stream, (const double *)w.partial, a.nchunks,
                          nprop, cst, logl);
  return launch_chained(noise_wv_const_kernel, (nprop + 255) / 256, 256, 0, stream, logl, nprop, cst);
}

int noise_bins_per_thread(int N, int nprop, int num_sms) {
  int R = kNoiseMaxBins;
  while (R > 1 && (long long)((N + kNoiseThreads * R - 1) / (kNoiseThreads * R)) * nprop <
                      (long long)kNoiseCtasPerSm * num_sms)
    R /= 2;
  return R;
}

// What any batch of at most nprop models needs: below the largest chunk the
// rule stops at the first size that reaches the target, at most twice it.
size_t noise_partials(int N, int nprop, int num_sms) {
  const int chunk = kNoiseThreads * kNoiseMaxBins;
  const size_t most = (size_t)nprop * ((N + chunk - 1) / chunk);
  const size_t few = 2 * (size_t)kNoiseCtasPerSm * num_sms + 2 * (size_t)nprop;
  return most > few ? most : few;
}

static size_t spline_smem(int nch, int kmax) { return sizeof(double) * (size_t)kmax * (1 + 6 * nch); }

cudaError_t spline_noise_launch(const SplineNoiseDev &s, int nprop, int kmax, const int *nknots, const double *knot_f,
                                const double *knot_C, double *logl, cudaStream_t stream, int *nlaunch) {
  static LaunchSetup setup;
  int dummy = 0;
  cudaError_t e = launch_setup(setup, [&](int *o) {
    *o = 1;
    return cudaFuncSetAttribute(spline_noise_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)spline_smem(2, kSplineMaxKnots));
  }, &dummy);
  if (e != cudaSuccess) return e;
  SplineNoiseArgs a;
  a.nch = s.nch;
  a.N = s.N;
  a.kmax = kmax;
  a.tab = s.tab;
  a.nknots = nknots;
  a.knot_f = knot_f;
  a.knot_C = knot_C;
  a.logl = logl;
  spline_noise_kernel<<<nprop, kSplineThreads, spline_smem(s.nch, kmax), stream>>>(a);
  if (nlaunch) *nlaunch = 1;
  return cudaGetLastError();
}

cudaError_t noise_logl_launch(const NoiseDev &nd, int nprop, const double *inst, const double *sgal, int sg_type,
                              const double *sgwb, double *logl, int num_sms, cudaStream_t stream, int *nlaunch) {
  NoiseArgs a;
  a.N = nd.N;
  a.R = noise_bins_per_thread(nd.N, nprop, num_sms);
  a.nchunks = (nd.N + kNoiseThreads * a.R - 1) / (kNoiseThreads * a.R);
  a.fstep = kNoiseThreads / nd.T;
  a.nprop = nprop;
  a.tab = nd.tab;
  a.inst = inst;
  a.sgal = sgal;
  a.sg_type = sg_type;
  a.sgwb = sgwb;
  a.rsg = nd.rsg;
  a.partial = nd.partial;
  int launches = 0;
  // models in slices of at most 65535 (the grid's y extent)
  for (int p0 = 0; p0 < nprop; p0 += 65535) {
    const int np = nprop - p0 < 65535 ? nprop - p0 : 65535;
    NoiseArgs s = a;
    s.nprop = np;
    s.inst = inst + 12 * (size_t)p0;
    s.sgal = sgal ? sgal + 5 * (size_t)p0 : nullptr;
    s.sgwb = sgwb ? sgwb + 4 * (size_t)p0 : nullptr;
    s.partial = nd.partial + (size_t)p0 * a.nchunks;
    const cudaError_t e =
        nd.nch == 3 ? launch_chained(noise_logl_kernel, dim3(a.nchunks, np), kNoiseThreads, 0, stream, s)
                    : launch_chained(noise_ch12_kernel, dim3(a.nchunks, np), kNoiseThreads, 0, stream, s, nd.nch);
    launches++;
    if (e != cudaSuccess) return e;
  }
  const double cst = nd.nch == 3 ? 3 * nd.N * log(2 * M_PI) : 0.0;
  launches++;
  if (nlaunch) *nlaunch = launches;
  return launch_chained(noise_finish_kernel, (nprop + 255) / 256, 256, 0, stream, (const double *)nd.partial, a.nchunks,
                        nprop, cst, logl);
}

}  // namespace glass
