// Fourier-domain UCB waveform and delta-logL kernels for sm_103a: plan,
// tables, orchestration and the drop-in single-waveform path.
//
// The reference computes one template at a time on the CPU: ucb_waveform
// (ucb/src/glass_ucb_waveform.c:738-1001) evaluates the slowly varying part of
// the response of the six LISA arms at N sample times, takes six N-point FFTs,
// and synthesises the TDI channels bin by bin (utils/src/glass_lisa.c:645-710);
// gaussian_log_likelihood (utils/src/glass_model.c:726-774) then sums the
// noise-weighted residual power over the whole segment.
//
// Here a batch of proposals of mixed sizes N (32..4096) is evaluated in three
// steps on one stream:
//   1. plan (FP64, spread over warps): the reference's bandwidth rule
//      gives N, the alignment gives the template's first segment bin, and the
//      per-proposal constants are prepared; proposals are binned by N;
//   2. slow part (one thread per (proposal, sample), all sizes in one launch):
//      the six arm responses, combined in the time domain into the four series
//      whose FFTs make the A and E channels (the TDI sums are linear, so
//      FFT(a - b) replaces FFT(a) - FFT(b)); written to an L2-resident scratch;
//   3. per size, concurrently: four N-point radix-4/2 Stockham FFTs in shared
//      memory, the per-segment-bin table folding TDI transfer factors, the A/E
//      combination and noise whitening, and the residual power over the
//      template support reduced to one number per proposal.
// Only the template support is visited: logL(r - h) - logL(r) differs from zero
// only there.
//
// Two precisions share the structure: plain FP64 (this file and
// ucb_fd_fp64.cu; the delay and carrier phase round each operation on its
// own, as the reference's C does), and a mixed form
// (ucb_fd_mixed.cu) in which the carrier phase is carried in double-float
// arithmetic and everything else is FP32.
#include "ucb_fd_device.cuh"

namespace glass {

cudaError_t fd_launch_slow_mixed(const SlowArgs &a, int num_sms, cudaStream_t stream, int block, int cap);
cudaError_t fd_launch_slow_fp64(const SlowArgs &a, int num_sms, cudaStream_t stream);
cudaError_t fd_launch_spec_mixed(int N, const SpecArgs &a, int nitems, int num_sms, cudaStream_t stream, bool perch);
cudaError_t fd_launch_spec_fp64(int N, const SpecArgs &a, int nitems, int num_sms, cudaStream_t stream, bool perch);
cudaError_t fd_launch_spec_all_mixed(const SpecAllArgs &A, int num_sms, cudaStream_t stream, bool perch, int cap);
cudaError_t fd_launch_spec_all_fp64(const SpecAllArgs &A, int num_sms, cudaStream_t stream, bool perch);
cudaError_t fd_launch_spec_cluster_fp64(const SpecSmallArgs &A, cudaStream_t stream, bool perch);

// ------------------------------------------------------------- plan kernel
// The two spreads of the bandwidth rule (ucb/src/glass_ucb_waveform.c:708-722, with
// AEnoise, utils/src/glass_lisa.c:1188-1198) in FP64, evaluated with one sincos and
// products: sin(acos(c)) as sqrt((1 - c)(1 + c)), x^10 as ((x^2)^2)^2 x^2, cos 2x as
// 2 cos^2 x - 1.  These agree with the library forms to a few ulp, so N can
// differ from the reference's only for a spread within ~1e-15 of a power of
// two (where the reference's own result depends on its libm).
__device__ __noinline__ int doppler_spread_fp64(double T, double f0, double fdot, double costheta) {
  const double sintheta = sqrt((1.0 - costheta) * (1.0 + costheta));
  return pow2_above_dev(2 * T * ((4. + kPI2 * f0 * (kAU / kCLIGHT) * sintheta) * (1.0 / kYEAR) + fabs(fdot) * T) - 1);
}
__device__ __noinline__ int snr_spread_fp64(const PlanArgs &a, double f0, double lnA) {
  double sf, cf;
  sincos_tab(div_by(f0, a.fstar, a.invfstar), a.tw1024, &sf, &cf);
  const double rf = rcp_fast(f0), r = 1.0e-4 * rf, q = 2.0e-5 * rf, q2 = q * q, q4 = q2 * q2;
  const double red = 1. + 16.0 * (q4 * q4 * q2 + r * r);
  const double rw = rf * (1.0 / kPI2), rw2 = rw * rw;
  const double c2x = 2.0 * cf * cf - 1.0;
  const double sn4L2 = (16.0 / 3.0) * sf * sf *
                       ((2.0 + cf) * (kSPS + kSLOC) + 2.0 * (3.0 + 2.0 * cf + c2x) * (kSLOC / 2.0 + kSACC * (rw2 * rw2) * red));
  return pow2_above_dev(exp(lnA) * sqrt(a.T) * sf * (2.0 * a.L) / sqrt(sn4L2) - 1);
}

// The bandwidth rule of ucb/src/glass_ucb_waveform.c:698-725: N is always the
// reference's.  A spread is evaluated in FP64 only where its FP32 interval leaves
// N open, which one proposal in 20,000 does; that lane runs 100 FP64
// instructions, while its CTA waits.
__device__ __forceinline__ int plan_size(const PlanArgs &a, const double *p, double f0) {
  SpreadInterval s = spread_interval(a.T, a.invfstar, a.L, a.NFFT, f0, p[1], to_f32(p[3]), to_f32(p[7]));
  if (s.open() && s.D0 != s.D1) {
    const int D = doppler_spread_fp64(a.T, f0, div_by(p[7], a.T2, a.invT2), p[1]);
    s.D0 = s.D1 = s.clamp(D);
  }
  if (s.open()) s.S0 = s.clamp(snr_spread_fp64(a, f0, p[3]));
  return 2 * max(s.D0, s.S0);
}

// Warp-aggregated binning: one atomic per distinct size per warp, begun by
// bin_begin, which returns its result to the group's first lane, and the list
// entries written by bin_end (so that the atomic's round trip passes behind other
// work).
struct BinSlot {
  unsigned same;
  int base;
};
__device__ __forceinline__ BinSlot bin_begin(const PlanArgs &a, int b) {
  BinSlot s = {__match_any_sync(0xffffffffu, b), 0};
  if (b >= 0 && (int)(threadIdx.x & 31) == __ffs(s.same) - 1) s.base = atomicAdd(&a.bin_count[b], __popc(s.same));
  return s;
}
__device__ __forceinline__ void bin_end(const PlanArgs &a, const BinSlot &s, int i, int b) {
  const int lane = threadIdx.x & 31, base = __shfl_sync(0xffffffffu, s.base, __ffs(s.same) - 1);
  const int slot = base + __popc(s.same & ((1u << lane) - 1));
  if (b >= 0 && chk(slot < a.cap && b < kNumBins, kChkBinList)) a.bin_list[(size_t)b * a.cap + slot] = i;
}

// u (component r of the sky basis vector along theta) and v (along phi).
__device__ __forceinline__ double sky_u(int r, double cth, double sth, double sph, double cph) {
  return r == 2 ? -sth : cth * (r == 0 ? cph : sph);
}
__device__ __forceinline__ double sky_v(int r, double sph, double cph) { return r == 2 ? 0.0 : (r == 0 ? sph : -cph); }

// Plan: size and placement of each proposal's template, its constants in the
// record of the path that follows, and its entry in its size's list.
//
// Latency-bound on FP64: an FP64 instruction, or a conversion to or from FP64,
// occupies a sub-partition for 64 clocks whatever the number of active lanes and
// of independent ones behind it, so the time is that of the warp with the most
// of them.  The work of P proposals is therefore spread over the four warps of
// a CTA (first part: warp 0 the sines and carrier constants, phi and 2 psi side
// by side in one warp's lanes; warp 1 size and placement, in FP32 up to the rule's
// boundaries; warp 2 amplitude and sine of theta; warp 3 the frequency constants)
// and, after a barrier, over all threads (second part: a tensor element each);
// quotients come from reciprocals of the batch's constants (correctly rounded),
// sines from the table, hi + lo floats and powers of two by integer arithmetic.
// P = ceil(n / SMs), 16 .. 32, keeps a batch of a few thousand on one wave.
// One proposal in FP64 23.6 -> 8.6 us, 3072 mixed 14.9 -> 10.4 us, 4096 for gradients
// 30 -> 14.2 us.
template <PlanKind KIND>
__global__ void __launch_bounds__(128) fd_plan_kernel(PlanArgs a) {
  __shared__ double2 s_sc[2][32];  // sine, cosine of phi and of 2 psi
  __shared__ double s_sth[32], s_amp[32], s_cthsth[32];
  __shared__ int s_st[32], s_N[32];
  __shared__ double s_p[32][9];  // parameters, rows of 9 against bank conflicts
  grid_begin();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, P = a.per_cta;
  const int i0 = blockIdx.x * P, n = min(P, a.nitems - i0);
  const int i = i0 + l;
  // one trip for all of a CTA's inputs, which may be pinned host memory that
  // changes between two replays of a graph: read through (ld.cv)
  int seg = -1;
  if (w == 1 && l < n) seg = __ldcv(a.item_seg + i);
  if (w == 2 && l < n && a.term_x_dev) a.term_x_dev[i] = __ldcv(a.term_x + i);
  for (int q = threadIdx.x; q < 8 * n; q += 128) s_p[q >> 3][q & 7] = __ldcv(a.params + 8 * (size_t)i0 + q);
  __syncthreads();
  const double *const p = s_p[l];
  ItemMix *const m = KIND == kPlanGrad ? &a.itemsgrad[l < n ? i : i0].m : a.itemsmix + (l < n ? i : i0);
  ItemF64 *const c64 = a.items64 + (l < n ? i : i0);
  if (w == 0) {
    for (int q = l; q < 2 * n; q += 32) {
      const int t = q >= n, j = t ? q - n : q;
      const double *pj = s_p[j];
      const double x = t ? 2. * pj[5] : pj[2];
      double s, c;
      sincos_tab(x, a.tw1024, &s, &c);
      s_sc[t][j] = make_double2(s, c);
    }
    if (l < n) {
      const double f0 = div_by(p[0], a.T, a.invT), fT = f0 * a.T;
      const double q = trunc_i64(fT);
      if (KIND == kPlanF64) {
        c64->f0 = f0;
        c64->dfq = kPI2 * div_by(q, a.T, a.invT);
        c64->phi0 = p[6];
      } else {
        split_f32(kPI2 * (fT - q), m->eps2pi.hi, m->eps2pi.lo);
        split_f32(p[6], m->phi0.hi, m->phi0.lo);
      }
    }
  } else if (w == 1) {
    if (l < n) {
      double v[8];
      int st = 0;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        v[k] = p[k];
        const unsigned long long b = (unsigned long long)__double_as_longlong(v[k]) << 1;  // |v|
        if (b >= 0x7ffull << 53) st = 1;                                                   // infinite or NaN
        if ((k == 1 || k == 4) && b > 0x3ffull << 53) st = 1;                              // |cosine| > 1
      }
      if (seg < 0 || seg >= a.nseg) st |= 2;
      int N = 0, imin = 0;
      if (!st) {
        const double f0 = div_by(v[0], a.T, a.invT);
        N = a.n_fixed > 0 ? a.n_fixed : plan_size(a, v, f0);
        if (N < kMinN || N > kMaxN) {
          st = 1;
        } else {
          imin = (int)((long long)(f0 * a.T) - N / 2) - a.seg_qmin[seg];
          if (imin >= a.NFFT || imin + N <= 0) st = 4;
        }
      }
      s_st[l] = st;
      s_N[l] = N;
      const int4 head = make_int4(seg, N, imin, 0);
      if (st)
        plan_write_skipped(a, i, st);
      else if (KIND == kPlanF64)
        c64->seg = head.x, c64->N = head.y, c64->imin = head.z, c64->pad = 0;
      else
        m->seg = head.x, m->N = head.y, m->imin = head.z, m->pad = 0;
    }
  } else if (w == 2) {
    if (l < n) {
      s_amp[l] = exp(p[3]);
      const double cth = p[1], sth = sqrt(fma(-cth, cth, 1.0));
      s_sth[l] = sth;
      if (KIND == kPlanGrad) s_cthsth[l] = cth / (sth < 1e-9 ? 1e-9 : sth);  // d/dcos(theta) is singular at the poles
    }
  } else if (l < n) {
    const double f0 = div_by(p[0], a.T, a.invT);
    if (KIND == kPlanF64) {
      const double fdot = div_by(p[7], a.T2, a.invT2);
      c64->w0 = kPI2 * f0;
      c64->wd = kPI * fdot;
      c64->ae = 0.66666666666666666666 * fdot / f0;
      c64->h0 = div_by(0.5 * f0, a.fstar, a.invfstar);
      c64->hd = div_by(0.5 * fdot, a.fstar, a.invfstar);
    } else {
      const double fdotT = div_by(p[7], a.T, a.invT);
      split_f32(div_by(f0, a.fstar, a.invfstar), m->fonfs0, m->fonfs0l);
      split_f32(div_by(fdotT, a.fstar, a.invfstar), m->fdfs, m->fdfsl);
      split_f32(0.66666666666666666666 * fdotT / f0, m->aef, m->aefl);
      split_f32(div_by(kPI2 * f0, kCLIGHT, a.invc), m->w0c, m->w0cl);
      split_f32(kPI * p[7], m->p7pi_d.hi, m->p7pi_d.lo);
      m->p7pi = m->p7pi_d.hi;
      if (KIND == kPlanGrad) {
        ItemGrad &g = a.itemsgrad[i];
        g.f0 = to_f32(f0);
        g.fdot = to_f32(div_by(p[7], a.T2, a.invT2));
        g.invT = to_f32(a.invT);
        g.fstar = to_f32(a.fstar);
      }
    }
  }
  __syncthreads();
  const int bin = w == 1 && l < n && s_st[l] == 0 ? fd_bin_of(s_N[l]) : -1;
  BinSlot slot = {0, 0};
  if (w == 1) slot = bin_begin(a, bin);
  for (int q = threadIdx.x; q < (KIND == kPlanF64 ? 2 : 8) * n; q += 128) {
    const int role = q / n, j = q - role * n;
    if (s_st[j]) continue;
    const double *pj = s_p[j];
    const double cth = pj[1], ci = pj[4], sth = s_sth[j];
    const double sph = s_sc[0][j].x, cph = s_sc[0][j].y, s2 = s_sc[1][j].x, c2 = s_sc[1][j].y;
    const double amp = scale_pow2(s_amp[j], -(32 - __clz(s_N[j])));  // amp / (2N), N a power of two
    if (KIND == kPlanF64) {
      ItemF64 &c = a.items64[i0 + j];
      if (role == 0) {
#pragma unroll
        for (int r = 0; r < 3; r++) {
          c.u[r] = sky_u(r, cth, sth, sph, cph);
          c.v[r] = sky_v(r, sph, cph);
        }
        c.k[0] = -sth * cph;
        c.k[1] = -sth * sph;
        c.k[2] = -cth;
      } else {
        const double Ap = (1. + ci * ci) * 0.5;
        c.DPr = Ap * c2;
        c.DPi = ci * s2;
        c.DC2r = 2.0 * (-Ap * s2);
        c.DC2i = 2.0 * (ci * c2);
        c.amp_s = amp;
      }
      continue;
    }
    ItemGrad *const g = KIND == kPlanGrad ? a.itemsgrad + i0 + j : nullptr;
    ItemMix &c = KIND == kPlanGrad ? g->m : a.itemsmix[i0 + j];
    const double Ap = (1. + ci * ci) * 0.5;
    if (role < 6) {
      // tensor element (r, s) of xx, xy, xz, yy, yz, zz.  amp/(2N) = msc 2^e, msc in
      // [1, 2): the power of two scales the template exactly in the likelihood
      // kernels, msc goes into the antenna tensors
      const int r = role < 3 ? 0 : (role < 5 ? 1 : 2), s = role < 3 ? role : (role < 5 ? role - 2 : 2);
      double ur = sky_u(r, cth, sth, sph, cph), us = sky_u(s, cth, sth, sph, cph);
      const double vr = sky_v(r, sph, cph), vs = sky_v(s, sph, cph);
      double ep = vr * vs - ur * us, ec = ur * vs + vr * us;
      int ex = ((__double2hiint(amp) >> 20) & 0x7ff) - 1023;
      if (ex <= -1023 || ex > 1023) ex = ilogb(amp);
      const double msc = scale_pow2(amp, -ex);
      split_f32(msc * (Ap * c2 * ep + -Ap * s2 * ec), c.Mr[role], c.Mrl[role]);
      split_f32(msc * (ci * s2 * ep + ci * c2 * ec), c.Mi[role], c.Mil[role]);
      if (role == 0) {
        c.amp_p2 = to_f32(scale_pow2(1.0, ex));
        split_f32(amp, c.amp_hi, c.amp_lo);
      }
      if (KIND == kPlanGrad) {
        // the tensors and their derivatives by cos(theta) and phi, at least 1e-9
        // from the poles
        if (sth < 1e-9) {
          ur = sky_u(r, cth, 1e-9, sph, cph);
          us = sky_u(s, cth, 1e-9, sph, cph);
          ep = vr * vs - ur * us;
          ec = ur * vs + vr * us;
        }
        const double uc[3] = {cph, sph, s_cthsth[j]};
        const double ucr = r == 0 ? uc[0] : (r == 1 ? uc[1] : uc[2]), ucs = s == 0 ? uc[0] : (s == 1 ? uc[1] : uc[2]);
        const double upr = r == 2 ? 0.0 : cth * (r == 0 ? -sph : cph), ups = s == 2 ? 0.0 : cth * (s == 0 ? -sph : cph);
        const double vpr = r == 2 ? 0.0 : (r == 0 ? cph : sph), vps = s == 2 ? 0.0 : (s == 0 ? cph : sph);
        g->ep[role] = to_f32(ep);
        g->ec[role] = to_f32(ec);
        g->dep_c[role] = to_f32(-ucr * us - ur * ucs);
        g->dec_c[role] = to_f32(ucr * vs + vr * ucs);
        g->dep_p[role] = to_f32(vpr * vs + vr * vps - upr * us - ur * ups);
        g->dec_p[role] = to_f32(upr * vs + ur * vps + vpr * us + vr * ups);
      }
    } else if (role == 6) {
      const double kx = -sth * cph, ky = -sth * sph;
      split_f32(kx, c.k[0], c.kl[0]);
      split_f32(ky, c.k[1], c.kl[1]);
      split_f32(-cth, c.k[2], c.kl[2]);
      c.k[3] = 0.f;
      const double bscale = kPI2 * div_by(pj[0], a.T, a.invT) * (kAU / kCLIGHT);
      split_f32(bscale * kx, c.beta1.hi, c.beta1.lo);
      split_f32(bscale * ky, c.beta2.hi, c.beta2.lo);
    } else if (KIND == kPlanGrad) {
      const double t = s_cthsth[j], sg = sth < 1e-9 ? 1e-9 : sth;
      g->dk_c[0] = to_f32(t * cph);
      g->dk_c[1] = to_f32(t * sph);
      g->dk_c[2] = -1.f;
      g->dk_c[3] = 0.f;
      g->dk_p[0] = to_f32(sg * sph);
      g->dk_p[1] = to_f32(-sg * cph);
      g->dk_p[2] = g->dk_p[3] = 0.f;
      const float ac = to_f32(Ap * c2), as = to_f32(Ap * s2), cc = to_f32(ci * c2), cs = to_f32(ci * s2);
      g->DP[0] = ac;
      g->DP[1] = cs;
      g->DC[0] = -as;
      g->DC[1] = cc;
      g->dDP_i[0] = cc;
      g->dDP_i[1] = to_f32(s2);
      g->dDC_i[0] = -cs;
      g->dDC_i[1] = to_f32(c2);
      g->dDP_s[0] = -2.f * as;
      g->dDP_s[1] = 2.f * cc;
      g->dDC_s[0] = -2.f * ac;
      g->dDC_s[1] = -2.f * cs;
    }
  }
  if (w == 1) {
    __syncwarp();
    bin_end(a, slot, i, bin);
  }
}

cudaError_t fd_launch_plan(PlanKind kind, PlanArgs a, const FdTablesDev &tab, int per_cta, int num_sms,
                           cudaStream_t stream) {
  const int per = num_sms > 0 ? (a.nitems + num_sms - 1) / num_sms : 16;
  a.per_cta = per_cta > 0 ? per_cta : (per < 16 ? 16 : (per > 32 ? 32 : per));
  a.invT = 1.0 / a.T;
  a.T2 = a.T * a.T;
  a.invT2 = 1.0 / a.T2;
  a.invfstar = 1.0 / a.fstar;
  a.invc = 1.0 / kCLIGHT;
  a.tw1024 = tab.tw64[fd_bin_of(kSincosTab)];
  const int grid = (a.nitems + a.per_cta - 1) / a.per_cta;
  switch (kind) {
    case kPlanF64: return launch_chained(fd_plan_kernel<kPlanF64>, grid, 128, 0, stream, a);
    case kPlanMix: return launch_chained(fd_plan_kernel<kPlanMix>, grid, 128, 0, stream, a);
    default: return launch_chained(fd_plan_kernel<kPlanGrad>, grid, 128, 0, stream, a);
  }
}

// Sets a CUDA-graph conditional node's value to (*count > 0).
__global__ void fd_cond_kernel(const int *count, cudaGraphConditionalHandle h) {
  if (threadIdx.x == 0) cudaGraphSetConditional(h, *(volatile const int *)count > 0 ? 1u : 0u);
}

// ------------------------------------------------------------ orbit tables
// One thread per (size, sample): analytic orbits of utils/src/glass_lisa.c:77-124
// at t = t0 + T (n-1)/N (ucb/src/glass_ucb_waveform.c:843), and the FFT
// twiddles exp(-2 pi i k / N).
__global__ void fd_orbit_table_kernel(FdTablesDev tab, double T, double t0) {
  int gid = blockIdx.x * blockDim.x + threadIdx.x;
  // sizes 32..4096 laid out back to back: offset of size b is 32 (2^b - 1)
  int b = 0;
  while (b < kNumBins && gid >= 32 * ((1 << (b + 1)) - 1)) b++;
  if (b >= kNumBins) return;
  int N = 32 << b;
  int n = gid - 32 * ((1 << b) - 1);
  double t = t0 + T * (double)n / (double)N;
  double alpha = kPI2 * t / kYEAR;
  double sa, ca;
  sincos(alpha, &sa, &ca);
  double ecc = kLARM / (2.0 * kSQ3 * kAU);
  double R = kAU * ecc;
  double sa2 = sa * sa, ca2 = ca * ca, saca = sa * ca, AUca = kAU * ca, AUsa = kAU * sa;
  const double sbs[3] = {0.0, 0.866025403784439, -0.866025403784438};
  const double cbs[3] = {1.0, -0.5, -0.5};
  OrbitSample64 o;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double sb = sbs[i], cb = cbs[i];
    o.x[i] = AUca + R * (saca * sb - (1. + sa2) * cb);
    o.y[i] = AUsa + R * (saca * cb - (1. + ca2) * sb);
    o.z[i] = -kSQ3 * R * (ca * cb + sa * sb);
  }
  o.t = t;
  orbit_arms(o);
  tab.pos64[b][n] = o;
  OrbitSampleMix m;
  df u = df_from_double(t / T), cd = df_from_double(ca), sd = df_from_double(sa);
  m.u_hi = u.hi;
  m.u_lo = u.lo;
  m.ca_hi = cd.hi;
  m.ca_lo = cd.lo;
  m.sa_hi = sd.hi;
  m.sa_lo = sd.lo;
  m.pad0 = m.pad1 = 0.f;
  tab.mix[b][n] = m;
  // mixed slow-part geometry: offsets from the guiding centre and arm monomials
  // (absent from tables built for the FP64 path alone)
  if (tab.geo[b]) {
    double v[28];
    double d[3][3];
    for (int i = 0; i < 3; i++) {
      d[i][0] = R * (saca * sbs[i] - (1. + sa2) * cbs[i]);
      d[i][1] = R * (saca * cbs[i] - (1. + ca2) * sbs[i]);
      d[i][2] = -kSQ3 * R * (ca * cbs[i] + sa * sbs[i]);
      for (int q = 0; q < 3; q++) v[3 * i + q] = d[i][q];
    }
    const int arm[3][2] = {{0, 1}, {0, 2}, {1, 2}};
    for (int a = 0; a < 3; a++) {
      double r[3];
      for (int q = 0; q < 3; q++) r[q] = (d[arm[a][1]][q] - d[arm[a][0]][q]) / kLARM;
      double *mo = v + 9 + 6 * a;
      mo[0] = r[0] * r[0];
      mo[1] = 2.0 * r[0] * r[1];
      mo[2] = 2.0 * r[0] * r[2];
      mo[3] = r[1] * r[1];
      mo[4] = 2.0 * r[1] * r[2];
      mo[5] = r[2] * r[2];
    }
    v[27] = 0.0;
    GeoSampleMix gm, gl;
    for (int q = 0; q < 28; q++) {
      gm.f[q] = (float)v[q];
      gl.f[q] = (float)(v[q] - (double)gm.f[q]);
    }
    tab.geo[b][n] = gm;
    if (tab.geolo[b]) tab.geolo[b][n] = gl;
  }
  double s, cth;
  sincospi(-2.0 * (double)n / (double)N, &s, &cth);
  tab.tw64[b][n] = make_double2(cth, s);
  tab.tt64[b][n] = tan_form(cth, s);
  tab.tw32[b][n] = make_float2((float)cth, (float)s);
  if (tab.tw32x[b]) {
    const float ch = (float)cth, sh = (float)s;
    tab.tw32x[b][n] = make_float4(ch, sh, (float)(cth - (double)ch), (float)(s - (double)sh));
  }
}

cudaError_t fd_build_orbit_tables(FdTablesDev &tab, double T, double t0, cudaStream_t stream) {
  if (!tab.base) {
    size_t total = 0;
    for (int b = 0; b < kNumBins; b++) {
      int N = 32 << b;
      total += (size_t)N * (sizeof(OrbitSample64) + sizeof(OrbitSampleMix) + 2 * sizeof(GeoSampleMix) +
                            sizeof(float2) + 2 * sizeof(double2) + sizeof(float4));
    }
    cudaError_t e = cudaMalloc(&tab.base, total);
    if (e != cudaSuccess) return e;
    char *p = (char *)tab.base;
    for (int b = 0; b < kNumBins; b++) {
      int N = 32 << b;
      tab.pos64[b] = (OrbitSample64 *)p;
      p += (size_t)N * sizeof(OrbitSample64);
      tab.mix[b] = (OrbitSampleMix *)p;
      p += (size_t)N * sizeof(OrbitSampleMix);
      tab.geo[b] = (GeoSampleMix *)p;
      p += (size_t)N * sizeof(GeoSampleMix);
      tab.geolo[b] = (GeoSampleMix *)p;
      p += (size_t)N * sizeof(GeoSampleMix);
      tab.tw64[b] = (double2 *)p;
      p += (size_t)N * sizeof(double2);
      tab.tt64[b] = (double2 *)p;
      p += (size_t)N * sizeof(double2);
      tab.tw32[b] = (float2 *)p;
      p += (size_t)N * sizeof(float2);
      tab.tw32x[b] = (float4 *)p;
      p += (size_t)N * sizeof(float4);
    }
  }
  int total = 32 * ((1 << kNumBins) - 1);
  fd_orbit_table_kernel<<<(total + 255) / 256, 256, 0, stream>>>(tab, T, t0);
  return cudaGetLastError();
}

// ---------------------------------------------------------- host: bank tables
void fd_build_bank_tables(int format, double T, double fstar, int NFFT, int nseg, const int *qmin, const double *rA,
                          const double *rE, const double *invCA, const double *invCE, float4 *w32, float4 *w32lo,
                          float4 *g32, double *Q, double2 *w64, double2 *g64, double *QA, float4 *g32lo) {
  const double sqT = sqrt(T);
  for (int s = 0; s < nseg; s++) {
    double q = 0.0, qa = 0.0;
    Q[(size_t)s * (NFFT + 1)] = 0.0;
    if (QA) QA[(size_t)s * (NFFT + 1)] = 0.0;
    for (int j = 0; j < NFFT; j++) {
      size_t sj = (size_t)s * NFFT + j;
      double f = (double)(qmin[s] + j) / T;
      double x = f / fstar;
      double c1 = cos(x), s1 = sin(x);
      double c2 = 2. * c1 * c1 - 1.0, s2 = 2. * s1 * c1;
      double c3 = 2. * c1 * c2 - c1, s3 = 2. * s1 * c2 + s1;
      double pref, w2r, w2i, w1r, w1i;
      if (format == 0) {  // sangria: utils/src/glass_lisa.c:685-700
        pref = f * (4.0 / fstar * sqT) * s1;
        w2r = c2; w2i = -s2;
        w1r = c1; w1i = -s1;
      } else {  // phase (:480-530) / frequency (:574-630)
        pref = (format == 1) ? sqT : sqT * 2. * x;
        w2r = c3 - c1; w2i = -s3 + s1;
        w1r = c2 - 1.0; w1i = -s2;
      }
      double sA = sqrt(invCA[sj]), sE = sqrt(invCE[sj]);
      double ka = sA * kSQRT1_2 * pref, ke = sE * kINVSQ6 * pref;
      double GA2r = ka * w2r, GA2i = ka * w2i, GA1r = ka * w1r, GA1i = ka * w1i;
      double GE2r = ke * w2r, GE2i = ke * w2i, GE1r = ke * w1r, GE1i = ke * w1i;
      double conj = (format == 1) ? -1.0 : 1.0;  // "phase" conjugates A and E (:545-546)
      double wAr = rA[2 * sj] * sA, wAi = conj * rA[2 * sj + 1] * sA;
      double wEr = rE[2 * sj] * sE, wEi = conj * rE[2 * sj + 1] * sE;
      w64[2 * sj] = make_double2(wAr, wAi);
      w64[2 * sj + 1] = make_double2(wEr, wEi);
      g64[4 * sj + 0] = make_double2(GA2r, GA2i);
      g64[4 * sj + 1] = make_double2(GA1r, GA1i);
      g64[4 * sj + 2] = make_double2(GE2r, GE2i);
      g64[4 * sj + 3] = make_double2(GE1r, GE1i);
      // The whitened data of a loud source reach |w| ~ 50 in its bins; rounded
      // to float, their cross term with the template would carry ~1e-3 of
      // error into delta logL, so the residual is kept as a double-float pair.
      float4 wf = make_float4((float)wAr, (float)wAi, (float)wEr, (float)wEi);
      w32[sj] = wf;
      w32lo[sj] = make_float4((float)(wAr - (double)wf.x), (float)(wAi - (double)wf.y), (float)(wEr - (double)wf.z),
                              (float)(wEi - (double)wf.w));
      const float4 ga = make_float4((float)GA2r, (float)GA2i, (float)GA1r, (float)GA1i);
      const float4 ge = make_float4((float)GE2r, (float)GE2i, (float)GE1r, (float)GE1i);
      g32[2 * sj] = ga;
      g32[2 * sj + 1] = ge;
      // a template's power sits in a few bins, so the rounding of these
      // entries would not average out over its support: kept as hi + lo
      if (g32lo) {
        g32lo[2 * sj] = make_float4((float)(GA2r - (double)ga.x), (float)(GA2i - (double)ga.y),
                                    (float)(GA1r - (double)ga.z), (float)(GA1i - (double)ga.w));
        g32lo[2 * sj + 1] = make_float4((float)(GE2r - (double)ge.x), (float)(GE2i - (double)ge.y),
                                        (float)(GE1r - (double)ge.z), (float)(GE1i - (double)ge.w));
      }
      q += wAr * wAr + wAi * wAi + wEr * wEr + wEi * wEi;
      Q[(size_t)s * (NFFT + 1) + j + 1] = q;
      if (QA) {
        qa += wAr * wAr + wAi * wAi;
        QA[(size_t)s * (NFFT + 1) + j + 1] = qa;
      }
    }
  }
}

// --------------------------------------------------------------- launchers
cudaError_t fd_dlogl_launch(const FdBankDev &bank, const FdTablesDev &tab, FdWorkDev &work, int precision,
                            int nitems, const int *item_seg, const double *params, const double *term_x,
                            double *dlogl, double *term_y, double *hh, int *status, int n_fixed, int num_sms,
                            cudaStream_t stream, int *nlaunch, double *term_ch, double *term_x_dev) {
  cudaError_t e;
  int launches = 0;
  const bool mix = precision == 1;
  if (!work.counts_zero) {
    e = cudaMemsetAsync(work.bin_count, 0, sizeof(int) * kFdCounts, stream);
    if (e != cudaSuccess) return e;
  }
  const bool fallback = mix && (work.fb_e1 > 0.f || work.fb_e2 > 0.f) && work.series2 != nullptr;
  work.counts_zero = false;  // until this sequence has been enqueued in full
  PlanArgs pa;
  pa.nitems = nitems;
  pa.nseg = bank.nseg;
  pa.NFFT = bank.NFFT;
  pa.cap = work.cap;
  pa.n_fixed = n_fixed;
  pa.T = bank.T;
  pa.fstar = bank.fstar;
  pa.L = kLARM;
  pa.item_seg = item_seg;
  pa.params = params;
  pa.term_x = term_x;
  pa.term_x_dev = term_x ? term_x_dev : nullptr;
  if (pa.term_x_dev) term_x = pa.term_x_dev;  // what the later kernels read
  pa.seg_qmin = bank.qmin;
  pa.items64 = work.items64;
  pa.itemsmix = work.itemsmix;
  pa.bin_count = work.bin_count;
  pa.bin_list = work.bin_list;
  pa.dlogl = dlogl;
  pa.term_y = term_y;
  pa.hh = hh;
  pa.status = status;
  const bool timing = work.phase_timing;
  work.phase_recorded = false;
  if (timing && (e = cudaEventRecord(work.phase[0], stream)) != cudaSuccess) return e;
  const int tune_per = work.tune.plan_per_cta;
  e = fd_launch_plan(mix ? kPlanMix : kPlanF64, pa, tab, tune_per >= 8 && tune_per <= 32 ? tune_per : 0, num_sms, stream);
  launches++;
  if (e != cudaSuccess) return e;
  if (timing && (e = cudaEventRecord(work.phase[1], stream)) != cudaSuccess) return e;

  SlowArgs sa;
  sa.cap = work.cap;
  sa.NFFT = bank.NFFT;
  sa.invLf = (float)(1.0 / kLARM);
  sa.AUcf = (float)(kAU / kCLIGHT);
  sa.invTf = (float)(1.0 / bank.T);
  sa.bin_count = work.bin_count;
  sa.bin_list = work.bin_list;
  sa.items64 = work.items64;
  sa.itemsmix = work.itemsmix;
  for (int b = 0; b < kNumBins; b++) {
    sa.pos64[b] = tab.pos64[b];
    sa.mix[b] = tab.mix[b];
    sa.geo[b] = tab.geo[b];
  }
  sa.tw1024 = tab.tw64[fd_bin_of(kSincosTab)];
  sa.series = work.series;
  sa.nitems = nitems;
  sa.series_len = (long long)(work.series_bytes / (mix ? sizeof(float2) : sizeof(double2)));
  e = mix ? fd_launch_slow_mixed(sa, num_sms, stream, work.tune.slow_block, work.tune.slow_ctas_per_sm)
          : fd_launch_slow_fp64(sa, num_sms, stream);
  launches++;
  if (e != cudaSuccess) return e;
  if (timing && (e = cudaEventRecord(work.phase[2], stream)) != cudaSuccess) return e;

  SpecArgs a;
  a.NFFT = bank.NFFT;
  a.cap = work.cap;
  a.bin_count = work.bin_count;
  a.items64 = work.items64;
  a.itemsmix = work.itemsmix;
  a.series = work.series;
  a.nitems = nitems;
  a.nseg = bank.nseg;
  a.series_len = sa.series_len;
  a.w32 = bank.w32;
  a.w32lo = bank.w32lo;
  a.g32 = bank.g32;
  a.g32lo = bank.g32lo;
  a.Q = bank.Q;
  a.w64 = bank.w64;
  a.g64 = bank.g64;
  a.term_x = term_x;
  a.dlogl = dlogl;
  a.term_y = term_y;
  a.hh = hh;
  a.status = status;
  a.term_ch = term_ch;
  a.QA = bank.QA;
  if (fallback) {
    a.fb_count = work.fb_count;
    a.hp_count = work.hp_count;
    a.hp_list = work.hp_list;
    a.fb_total = work.fb_total;
    a.fb_e1 = work.fb_e1;
    a.fb_e2 = work.fb_e2;
    a.fb_inv_scale = work.fb_inv_scale;
    a.fb_nscale = work.fb_nscale;
  }
  const bool perch = term_ch != nullptr;
  // Inside a CUDA-graph capture, the re-evaluation (two launches, idle in
  // batches with nothing listed) sits behind a conditional node that a
  // one-thread kernel sets when something is listed; outside capture, where
  // the graph API refuses, or for a batch so small that its two launches take
  // less than the node, it is launched unconditionally.
  bool cond = false;
  cudaGraphConditionalHandle cond_h = 0;
  cudaGraph_t cap_graph = nullptr;
  if (fallback && nitems > kSmallBatch) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamGetCaptureInfo(stream, &cs, nullptr, &cap_graph) == cudaSuccess &&
        cs == cudaStreamCaptureStatusActive &&
        cudaGraphConditionalHandleCreate(&cond_h, cap_graph, 0, cudaGraphCondAssignDefault) == cudaSuccess)
      cond = true;
    (void)cudaGetLastError();
  }
  // sizes up to 1024 (every size a segment of NFFT bins can produce, up to
  // NFFT: ucb_bandwidth caps N there) in one launch on the main stream; 2048
  // and 4096 as their own kernels on side streams running beside it
  int nall = 0;
  while (nall < kSpecAllBins && (32 << nall) <= bank.NFFT) nall++;
  int nb = 0;
  // a few FP64 proposals: a cluster of CTAs each, whatever the size (where the
  // line lies: at fd_spec_cluster64_kernel)
  const bool few = !mix && nall > 0 && nitems <= num_sms / 5;
  if (few) {
    SpecSmallArgs A;
    A.a = a;
    A.a.bin = 0;
    A.a.bin_list = work.bin_list;
    A.a.tw = nullptr;
    A.nbins = 0;
    for (int b = 0; b < kNumBins; b++) {
      A.tw[b] = tab.tt64[b];
      if (32 << b <= bank.NFFT) A.nbins = b + 1;
    }
    A.zero_counts = work.bin_count;
    A.done = work.bin_count + kNumBins + 1;
    e = fd_launch_spec_cluster_fp64(A, stream, perch);
    launches++;
    if (e != cudaSuccess) return e;
  }
  if (bank.NFFT > 1024 && !few) {
    if ((e = cudaEventRecord(work.fork, stream)) != cudaSuccess) return e;
    for (int b = kSpecAllBins; b < kNumBins; b++) {
      int N = 32 << b;
      if (N > bank.NFFT) break;
      cudaStream_t sb = work.side[b];
      if ((e = cudaStreamWaitEvent(sb, work.fork, 0)) != cudaSuccess) return e;
      a.bin = b;
      a.bin_list = work.bin_list + (size_t)b * work.cap;
      a.tw = mix ? (const void *)tab.tw32x[b] : (const void *)tab.tt64[b];
      e = mix ? fd_launch_spec_mixed(N, a, nitems, num_sms, sb, perch)
              : fd_launch_spec_fp64(N, a, nitems, num_sms, sb, perch);
      launches++;
      if (e != cudaSuccess) return e;
      if ((e = cudaEventRecord(work.join[b], sb)) != cudaSuccess) return e;
      nb++;
    }
  }
  if (nall > 0 && !few) {
    SpecAllArgs A;
    A.a = a;
    A.a.bin = 0;
    A.a.bin_list = work.bin_list;
    A.a.tw = nullptr;
    A.nbins = nall;
    A.zero_counts = nb == 0 ? work.bin_count : nullptr;  // side kernels would still be reading them
    A.done = work.bin_count + kNumBins + 1;  // fb_count is at kNumBins
    // In a graph a chained launch starts ahead of the size kernels on its side
    // branches, which suits a light batch (1000 proposals of at most 1024 points on
    // 2048 bins 35 -> 29 us) but not a large one whose size kernels end it, as with the
    // re-evaluation off: 10000 of up to 2048 points 1063 us after an ordinary launch,
    // 1115 chained, 3000 343 and 361; 3000 light ones 45.6 and 43.5.
    if (nb > 0 && mix && !fallback && nitems > 1024) {
      cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
      if ((e = cudaStreamIsCapturing(stream, &cs)) != cudaSuccess) return e;
      A.chained = cs != cudaStreamCaptureStatusActive;
    }
    for (int b = 0; b < kSpecAllBins; b++) A.tw[b] = mix ? (const void *)tab.tw32x[b] : (const void *)tab.tt64[b];
    e = mix ? fd_launch_spec_all_mixed(A, num_sms, stream, perch, work.tune.spec_ctas_per_sm)
            : fd_launch_spec_all_fp64(A, num_sms, stream, perch);
    launches++;
    if (e != cudaSuccess) return e;
  }
  for (int b = kSpecAllBins; b < kSpecAllBins + nb; b++)
    if ((e = cudaStreamWaitEvent(stream, work.join[b], 0)) != cudaSuccess) return e;
  // the size counts only: fb_count follows them (the re-evaluation's first kernel
  // zeroes them where it runs in any case)
  const bool counts_left = nb > 0 || nall == 0;
  if (counts_left && (!fallback || cond)) {
    if ((e = cudaMemsetAsync(work.bin_count, 0, sizeof(int) * kNumBins, stream)) != cudaSuccess) return e;
  }
  if (timing && (e = cudaEventRecord(work.phase[3], stream)) != cudaSuccess) return e;

  // Re-evaluation of the listed mixed proposals in double-float: series
  // (into series2), spectral stage, results written over the mixed ones; the
  // re-evaluation's counts and fb_count end at zero.
  if (fallback) {
    int nmax = kMaxN;
    while (nmax > bank.NFFT) nmax >>= 1;
    SlowArgs sh = sa;
    sh.bin_count = work.hp_count;
    sh.bin_list = work.hp_list;
    sh.zero_counts = counts_left && !cond ? work.bin_count : nullptr;
    sh.series = work.series2;
    sh.series_len = (long long)(work.series_bytes / sizeof(float4));
    for (int b = 0; b < kNumBins; b++) sh.geolo[b] = tab.geolo[b];
    sh.invLd = df_from_double(1.0 / kLARM);
    sh.AUcd = df_from_double(kAU / kCLIGHT);
    sh.invTd = df_from_double(1.0 / bank.T);
    sh.invcd = df_from_double(1.0 / kCLIGHT);
    HpArgs h;
    h.NFFT = bank.NFFT;
    h.cap = work.cap;
    h.nitems = nitems;
    h.nseg = bank.nseg;
    h.series_len = sh.series_len;
    h.nmax = nmax;
    h.bin_count = work.hp_count;
    h.bin_list = work.hp_list;
    h.itemsmix = work.itemsmix;
    h.series = reinterpret_cast<const float4 *>(work.series2);
    h.zero_at = work.fb_count;  // fb_count, the done counters, the spares and hp_count
    h.nzero = kFdCounts - kNumBins;
    h.done = work.bin_count + kNumBins + 2;
    h.w32 = bank.w32;
    h.w32lo = bank.w32lo;
    h.g32 = bank.g32;
    h.g32lo = bank.g32lo;
    h.Q = bank.Q;
    h.QA = bank.QA;
    for (int b = 0; b < kNumBins; b++) h.tw32x[b] = tab.tw32x[b];
    h.term_x = term_x;
    h.dlogl = dlogl;
    h.term_y = term_y;
    h.hh = hh;
    h.term_ch = term_ch;
    h.status = status;
    cudaStream_t ts = stream;
    cudaGraphNode_t cnode = nullptr;
    if (cond) {
      fd_cond_kernel<<<1, 32, 0, stream>>>(work.fb_count, cond_h);
      launches++;
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      const cudaGraphNode_t *deps = nullptr;
      size_t nd = 0;
      cudaStreamCaptureStatus cs;
      cudaGraphNodeParams np = {};
      np.type = cudaGraphNodeTypeConditional;
      np.conditional.handle = cond_h;
      np.conditional.type = cudaGraphCondTypeIf;
      np.conditional.size = 1;
      if ((e = cudaStreamGetCaptureInfo(stream, &cs, nullptr, nullptr, &deps, nullptr, &nd)) != cudaSuccess) return e;
      if ((e = cudaGraphAddNode(&cnode, cap_graph, deps, nullptr, nd, &np)) != cudaSuccess) return e;
      ts = work.side[0];
      if ((e = cudaStreamBeginCaptureToGraph(ts, np.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                             cudaStreamCaptureModeRelaxed)) != cudaSuccess)
        return e;
    }
    e = fd_launch_reeval(sh, h, perch, num_sms, ts, &launches);
    if (e != cudaSuccess) return e;
    if (cond) {
      cudaGraph_t body = nullptr;
      if ((e = cudaStreamEndCapture(ts, &body)) != cudaSuccess) return e;
      if ((e = cudaStreamUpdateCaptureDependencies(stream, &cnode, nullptr, 1, cudaStreamSetCaptureDependencies)) !=
          cudaSuccess)
        return e;
    }
  }
  work.counts_zero = true;
  if (timing) {
    if ((e = cudaEventRecord(work.phase[4], stream)) != cudaSuccess) return e;
    work.phase_recorded = true;
  }
  if (nlaunch) *nlaunch = launches;
  return cudaSuccess;
}

size_t fd_series_bytes(int nitems, int NFFT, int precision) {
  size_t elem = precision == 1 ? sizeof(float2) : sizeof(double2);
  return (size_t)nitems * (size_t)NFFT * 4 * elem;
}

// ------------------------------------------------------- legacy single waveform
// The drop-in ucb_waveform for one source: the per-source constants come from
// the host (source_geometry / make_item_f64, the same FP64 code); the six arm
// responses are computed one thread per sample spread over N/32 CTAs (the
// FP64 pipe of many SMs, not one); then one CTA per Michelson channel (X, Y,
// Z) FFTs its two series and applies the format's TDI weights per bin.  A and
// E follow in fd_ae_kernel from the stored X, Y, Z (utils/src/glass_lisa.c:429-441).
__global__ void fd_single_slow_kernel(const OrbitSample64 *pos, const ItemF64 *item, int N, const double2 *tw1024,
                                      double2 *d6) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  double2 d[6];
  slow_sample64(*item, pos[n], tw1024, d);
#pragma unroll
  for (int a = 0; a < 6; a++) d6[(size_t)a * N + n] = d[a];
}

template <int N>
struct LegacyCfg {
  static constexpr int R = (N <= 128) ? 4 : 8;  // bins per thread
  static constexpr int GT = N / R;              // threads (one CTA per channel)
};

template <int N>
__global__ void __launch_bounds__(LegacyCfg<N>::GT) fd_waveform_kernel(const ItemF64 *item, const double2 *d6,
                                                                    int format, double T, double fstar,
                                                                    double *out, const double2 *twg) {
  constexpr int GT = LegacyCfg<N>::GT, R = LegacyCfg<N>::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *tw = reinterpret_cast<double2 *>(smem_raw);
  double2 *buf = tw + N;
  const int lane = threadIdx.x, ch = blockIdx.x;
  for (int i = lane; i < N; i += GT) tw[i] = twg[i];
  // d: 12, 13, 21, 23, 31, 32 ; X: (12-13, 21-31), Y: (23-21, 32-12), Z: (31-32, 13-23)
  const int ua = ch == 0 ? 0 : ch == 1 ? 3 : 4, ub = ch == 0 ? 1 : ch == 1 ? 2 : 5;
  const int va = ch == 0 ? 2 : ch == 1 ? 5 : 1, vb = ch == 0 ? 4 : ch == 1 ? 0 : 3;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int n = lane + GT * r;
    buf[n] = csub(d6[(size_t)ua * N + n], d6[(size_t)ub * N + n]);
    buf[N + n] = csub(d6[(size_t)va * N + n], d6[(size_t)vb * N + n]);
  }
  __syncthreads();
  group_fft<N, GT, 2, 1, double2, true>(buf, tw, lane);  // CTA barrier: the CTA may be a partial warp
  const double sqT = sqrt(T);
  const long long q = (long long)(item->f0 * T);
  const double amp_s = item->amp_s;
  double *X = out + (size_t)ch * 2 * N;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = lane + GT * r;
    const int m = (k + N / 2) & (N - 1);
    double f = (double)(q + m - N / 2) / T;
    double x = f / fstar;
    double s1, c1;
    sincos(x, &s1, &c1);
    double c2 = 2. * c1 * c1 - 1.0, s2 = 2. * s1 * c1;
    double2 W2, W1;
    double pref;
    if (format == 0) {
      pref = f * (4.0 / fstar * sqT) * s1;
      W2 = make_double2(c2, -s2);
      W1 = make_double2(c1, -s1);
    } else {
      double c3 = 2. * c1 * c2 - c1, s3 = 2. * s1 * c2 + s1;
      pref = (format == 1) ? sqT : sqT * 2. * x;
      W2 = make_double2(c3 - c1, -s3 + s1);
      W1 = make_double2(c2 - 1.0, -s2);
    }
    double2 h = cadd(cmul(buf[k], W2), cmul(buf[N + k], W1));
    double sc = amp_s * pref;
    X[2 * m] = h.x * sc;
    X[2 * m + 1] = h.y * sc;
  }
}

__global__ void fd_ae_kernel(double *out, int N, int format) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= 2 * N) return;
  const double *X = out, *Y = out + 2 * N, *Z = out + 4 * N;
  double *A = out + 6 * N, *E = out + 8 * N;
  double a = (Z[m] - X[m]) * kSQRT1_2;
  double e = (X[m] - 2 * Y[m] + Z[m]) * kINVSQ6;
  if (format == 1 && (m & 1)) {
    a = -a;
    e = -e;
  }
  A[m] = a;
  E[m] = e;
}

template <int N>
static cudaError_t launch_waveform(const ItemF64 *item, const double2 *d6, int format, int nch, double T, double fstar,
                                   double *out, const double2 *tw, cudaStream_t stream) {
  size_t smem = sizeof(double2) * 3 * N;
  static LaunchSetup setup;
  int occ = 0;
  cudaError_t e = launch_setup(setup, [&](int *o) {
    *o = 1;
    return cudaFuncSetAttribute(fd_waveform_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }, &occ);
  if (e != cudaSuccess) return e;
  fd_waveform_kernel<N><<<nch, LegacyCfg<N>::GT, smem, stream>>>(item, d6, format, T, fstar, out, tw);
  return cudaGetLastError();
}

cudaError_t fd_waveform_launch(const OrbitSample64 *pos, const ItemF64 *item, int N, int format, int NI, double T,
                               double fstar, double2 *d6, double *out, const double2 *tw, const double2 *tw1024,
                               cudaStream_t stream) {
  int nch = (format != 0 && NI <= 1) ? 1 : 3;
  fd_single_slow_kernel<<<(N + 31) / 32, 32, 0, stream>>>(pos, item, N, tw1024, d6);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = cudaErrorInvalidValue;
  switch (N) {
#define GLASS_WCASE(NN) \
  case NN:              \
    e = launch_waveform<NN>(item, d6, format, nch, T, fstar, out, tw, stream); \
    break;
    GLASS_WCASE(32)
    GLASS_WCASE(64)
    GLASS_WCASE(128)
    GLASS_WCASE(256)
    GLASS_WCASE(512)
    GLASS_WCASE(1024)
    GLASS_WCASE(2048)
    GLASS_WCASE(4096)
#undef GLASS_WCASE
  }
  if (e != cudaSuccess) return e;
  if (nch == 3) {
    fd_ae_kernel<<<(2 * N + 127) / 128, 128, 0, stream>>>(out, N, format);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace glass
