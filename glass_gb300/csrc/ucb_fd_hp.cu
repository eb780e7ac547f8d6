// Double-float re-evaluation of mixed-precision proposals.
//
// The mixed path's template is an FP32 FFT of FP32 series from FP32
// per-proposal constants; its delta logL carries an error of up to
// ~6e-7 sqrt(hw rr / N) + 1.5e-7 |(h|r - h)| (whitened sums over the template
// support): below 1e-3 except for loud templates, near the data of a source
// with SNR ~ 300 or far from the data with (h|h) ~ 1e6.  The mixed spectral
// kernels estimate it and list those
// proposals by size, and they are evaluated again with every step in
// double-float arithmetic (pairs of floats, ~48 bits, on the FP32 pipe, which
// on GB300 runs 64 times the FP64 rate), in two launches:
//   fd_slow_hp_kernel: their four A/E arm-combination series in
//     double-float, three warps per 32 samples: the mixed slow part's formulation
//     (carrier phase heterodyned to the segment and reduced mod 2 pi, so that
//     its absolute error stays ~1e-12 rad) with every product and sum in
//     double-float, double-float sine, cosine (table of k pi/32 plus short
//     Taylor series) and sinc, and the per-sample
//     geometry and per-proposal constants as hi + lo floats;
//   fd_hp_kernel:      thread-block clusters of 4 CTAs, one proposal each:
//     CTA r transforms series r in place in its shared memory (radix 4,
//     twiddles as hi + lo floats), then CTAs 2c and 2c + 1 form channel c's
//     whitened template per bin from their own spectrum and their partner's
//     (read through distributed shared memory), each over half of the bins,
//     and sum the residual power and the template power; CTA 0 gathers the
//     four partial sums and writes the results over the mixed ones.  Proposals of
//     up to 256 points, and of 512 where clusters would queue, take one CTA each,
//     with the same sums.
// What is left is of order 1e-12 of the same scale.
#include <math.h>

#include <cooperative_groups.h>

#include "ucb_fd_device.cuh"

namespace glass {

constexpr int kHpThreads = 256;

// -------------------------------------------------------- slow part, df
// k.(x_i - x_gc) of spacecraft i (metres).
__device__ __forceinline__ df kdot_hp(const ItemMix &c, const GeoSampleMix &gm, const GeoSampleMix &gl, int i) {
  const df k0 = {c.k[0], c.kl[0]}, k1 = {c.k[1], c.kl[1]}, k2 = {c.k[2], c.kl[2]};
  return df_add(df_add(df_mul(k0, df{gm.f[3 * i], gl.f[3 * i]}), df_mul(k1, df{gm.f[3 * i + 1], gl.f[3 * i + 1]})),
                df_mul(k2, df{gm.f[3 * i + 2], gl.f[3 * i + 2]}));
}
// r^T M r of arm a (0: 12, 1: 13, 2: 23), M = m (DP e+ + DC ex) as hi + lo.
__device__ __forceinline__ dc arm_hp(const ItemMix &c, const GeoSampleMix &gm, const GeoSampleMix &gl, int a) {
  df mr = {0.f, 0.f}, mi = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < 6; t++) {
    const df mo = {gm.f[9 + 6 * a + t], gl.f[9 + 6 * a + t]};
    mr = df_add(mr, df_mul(df{c.Mr[t], c.Mrl[t]}, mo));
    mi = df_add(mi, df_mul(df{c.Mi[t], c.Mil[t]}, mo));
  }
  return {mr, mi};
}

// The two arms of spacecraft i (12, 13 | 21, 23 | 31, 32) at one sample, as
// slow_sample_mix computes them, in double-float throughout, from the three
// spacecraft's kdot_hp and the three arms' arm_hp.  tab: the sine/cosine table of
// df_sincos_tab.
__device__ __forceinline__ void slow_arms_hp(const ItemMix &c, const OrbitSampleMix &o, const df kd[3], const dc m[3],
                                             const SlowArgs &K, const float4 *tab, int i, dc d[2]) {
  const df k0 = {c.k[0], c.kl[0]}, k1 = {c.k[1], c.kl[1]};
  // this spacecraft's two arms as unique arms (0: 12, 1: 13, 2: 23) with the
  // orientation signs of k.r: 12 +0, 13 +1 | 21 -0, 23 +2 | 31 -1, 32 -2
  const int ua[2] = {i == 2 ? 1 : 0, i == 0 ? 1 : 2};
  const bool neg[2] = {i != 0, i == 2};
  const df psi0 = carrier_phase_mix(c, o);
  const df u = {o.u_hi, o.u_lo}, ca = {o.ca_hi, o.ca_lo}, sa = {o.sa_hi, o.sa_lo};
  const df tgc = df_mul(K.AUcd, df_add(df_mul(k0, ca), df_mul(k1, sa)));  // guiding-centre delay (s)
  const df tT = df_mul(df_add(tgc, df_mul(kd[i], K.invcd)), K.invTd);    // tau_i / T
  const df v = df_add(u, df_neg(tT));                                    // xi / T
  const df fon = df_add(df{c.fonfs0, c.fonfs0l}, df_mul(df{c.fdfs, c.fdfsl}, v));
  const df aev = df_add(df{1.f, 0.f}, df_mul(df{c.aef, c.aefl}, v));
  const df arg2 = df_add(df_add(psi0, df_neg(df_mul(df{c.w0c, c.w0cl}, kd[i]))),
                         df_mul(c.p7pi_d, df_mul(tT, df_add(tT, df{-2.f * u.hi, -2.f * u.lo}))));
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int a = ua[q];
    df kr = df_mul(df_add(kd[a == 0 ? 1 : 2], df_neg(kd[a == 2 ? 1 : 0])), K.invLd);
    if (neg[q]) kr = df_neg(kr);
    const df h1 = df_add(df{1.f, 0.f}, kr);
    const df arg1 = df_mul(df{0.5f * fon.hi, 0.5f * fon.lo}, h1);
    const df sc = df_sinc(arg1, tab);
    const df sinc = {0.25f * sc.hi, 0.25f * sc.lo};
    const df t1r = df_mul(aev, m[a].re), t1i = df_mul(aev, m[a].im);
    df s2, c2;
    df_sincos_tab(df_add(arg1, df_neg(arg2)), tab, &s2, &c2);
    const df re = df_add(df_mul(t1r, c2), df_mul(t1i, s2));
    const df im = df_add(df_mul(t1i, c2), df_neg(df_mul(t1r, s2)));
    d[q] = {df_mul(sinc, re), df_mul(sinc, im)};
  }
}

// One CTA of three warps per 32 consecutive samples of one binned proposal,
// grid-stride over all of them: warp i computes k.x of spacecraft i and the
// antenna pattern of arm i, shared with the other two, then the arms of
// spacecraft i (a third of the dependent chain of a sample each, on separate SM
// sub-partitions); warps 0 and 1 then form the A and E arm combinations of
// ae_combos in double-float.
// sin(k pi / 32), cos(k pi / 32) as hi + lo floats {s.hi, s.lo, c.hi, c.lo},
// k < 64: built once per device on the host (hp_sincos_table).
static __device__ float4 g_hp_sincos[64];

__global__ void __launch_bounds__(96) fd_slow_hp_kernel(SlowArgs a) {
  __shared__ dc s_d[6][32], s_m[3][32];
  __shared__ float2 s_kd[3][32];
  __shared__ float4 s_tab[64];
  grid_begin();
  // the batch's size counts, which the spectral stage has read for the last time
  if (a.zero_counts && blockIdx.x == 0 && threadIdx.x < kNumBins) a.zero_counts[threadIdx.x] = 0;
  int cs[kNumBins + 1];
  int acc = 0;
#pragma unroll
  for (int b = 0; b < kNumBins; b++) {
    cs[b] = acc;
    if ((32 << b) <= a.NFFT) acc += a.bin_count[b] << b;
  }
  cs[kNumBins] = acc;
  if ((int)blockIdx.x >= acc) return;
  if (threadIdx.x < 64) s_tab[threadIdx.x] = g_hp_sincos[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31, sc = threadIdx.x >> 5;
  float4 *series = reinterpret_cast<float4 *>(a.series);
#pragma unroll 1
  for (int ch = blockIdx.x; ch < acc; ch += gridDim.x) {
    int b = 0, cb = 0;
#pragma unroll
    for (int bb = 1; bb < kNumBins; bb++)
      if (ch >= cs[bb]) {
        b = bb;
        cb = cs[bb];
      }
    const int N = 32 << b;
    const int local = ch - cb;
    const int slot = local >> b;
    const int n = ((local & ((1 << b) - 1)) << 5) + lane;
    // checked build: an index outside its buffer is recorded and the chunk
    // computed from proposal 0 without being written (the CTA keeps its
    // barriers)
    const bool lok = chk(slot < a.cap, kChkReevalList);
    int item = lok ? a.bin_list[(size_t)b * a.cap + slot] : 0;
    const bool iok = chk(item >= 0 && item < a.nitems, kChkItem);
    if (!iok) item = 0;
    const long long o0 = ((long long)cb * 32 + (long long)slot * N) * 4 + n;
    const bool wok = lok && iok && chk(o0 >= 0 && o0 + 3LL * N < a.series_len, kChkSeriesWrite);
    const ItemMix &c = a.itemsmix[item];
    const GeoSampleMix &gm = a.geo[b][n], &gl = a.geolo[b][n];
    const df kx = kdot_hp(c, gm, gl, sc);
    s_kd[sc][lane] = make_float2(kx.hi, kx.lo);
    s_m[sc][lane] = arm_hp(c, gm, gl, sc);
    __syncthreads();
    df kd[3];
    dc m[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const float2 v = s_kd[q][lane];
      kd[q] = {v.x, v.y};
      m[q] = s_m[q][lane];
    }
    dc d2[2];
    slow_arms_hp(c, a.mix[b][n], kd, m, a, s_tab, sc, d2);
    s_d[2 * sc][lane] = d2[0];
    s_d[2 * sc + 1][lane] = d2[1];
    __syncthreads();
    if (sc < 2 && wok) {
      dc d[6];
#pragma unroll
      for (int q = 0; q < 6; q++) d[q] = s_d[q][lane];
      // d: 12, 13, 21, 23, 31, 32
      dc c0, c1;
      if (sc == 0) {
        c0 = dc_sub(dc_add(d[4], d[1]), dc_add(d[5], d[0]));  // a2
        c1 = dc_sub(dc_add(d[1], d[4]), dc_add(d[3], d[2]));  // a1
      } else {
        const dc t2 = dc_sub(d[2], d[3]), t1 = dc_sub(d[0], d[5]);
        c0 = dc_add(dc_sub(dc_sub(dc_add(d[0], d[4]), d[1]), d[5]), dc_add(t2, t2));  // e2
        c1 = dc_add(dc_sub(dc_sub(dc_add(d[1], d[2]), d[3]), d[4]), dc_add(t1, t1));  // e1
      }
      float4 *out = series + ((long long)cb * 32 + (long long)slot * N) * 4 + (size_t)(2 * sc) * N + n;
      out[0] = make_float4(c0.re.hi, c0.im.hi, c0.re.lo, c0.im.lo);
      out[N] = make_float4(c1.re.hi, c1.im.hi, c1.re.lo, c1.im.lo);
    }
    __syncthreads();
  }
}

// Proposals of up to 256 points (sizes b < kHpSmallBins, 32 << b) take one CTA each,
// those of 512 too where the clusters are too few and either every one finds a CTA
// beside the larger ones' clusters or the batch is several waves long.
constexpr int kHpSmallBins = 4;
constexpr int kHpSmallMax = 32 << kHpSmallBins;

// ------------------------------------------------------- spectral stage, df
// The proposal of entry k (largest sizes first, so that the long ones start
// early): item, size, segment, placement, size bin and series offset (float4
// elements).  cs[b]: the first entry of size bin b.
struct HpEntry {
  int item, N, seg, imin, bin;
  long long off;
  float amp_p2;
  bool ok;  // checked build: every index in bounds (else read safely, not written)
};

__device__ __forceinline__ HpEntry hp_entry(const HpArgs &a, int k, const int *cs) {
  int bin = kNumBins - 1;
#pragma unroll
  for (int b = kNumBins - 2; b >= 0; b--)
    if (k >= cs[b]) bin = b;
  const int slot = k - cs[bin];
  HpEntry e;
  e.ok = chk(slot < a.cap, kChkReevalList);
  e.item = e.ok ? a.bin_list[(size_t)bin * a.cap + slot] : 0;
  e.ok = e.ok && chk(e.item >= 0 && e.item < a.nitems, kChkItem);
  const ItemMix &c = a.itemsmix[e.ok ? e.item : 0];
  e.N = c.N;
  e.seg = c.seg;
  e.imin = c.imin;
  e.bin = bin;
  e.off = (bin_sample_start(a.bin_count, a.NFFT, bin) + (long long)slot * c.N) * 4;
  e.amp_p2 = c.amp_p2;
  e.ok = e.ok && chk(e.seg >= 0 && e.seg < a.nseg, kChkBankRead) &&
         chk(e.N >= 32 && e.N <= a.nmax && e.off >= 0 && e.off + 4LL * e.N <= a.series_len, kChkSeriesRead);
  if (!e.ok) {
    e.N = 32;
    e.bin = 0;
    e.seg = 0;
    e.off = 0;
  }
  return e;
}

// Latency-bound: a batch lists tens of proposals, each a chain of dependent loads,
// five or six FFT stages and cluster barriers, so what matters is that all of
// them are resident at once and that the chain is short.  In place and with the
// twiddles in L1 a CTA takes 16 bytes per point (64 KB at N = 4096, where
// ping-pong buffers and a twiddle copy took 192 KB and left one CTA per SM); the
// bank's entries of a thread's first bins are loaded before the transform, those
// of each next bin and the twiddles of each next butterfly before the arithmetic of
// the current one.  61 proposals of up to 1024 points 19.1 -> 16 us, 73 of up to
// 4096 on 8192-bin segments 60.8 -> 36 us.
//
// The registers that takes leave 74 clusters resident.  Up to 256 points one CTA
// holds a proposal's four series and has a butterfly of a stage per thread, as
// a cluster has, without its barriers: 296 at once (series and transform of 3000
// proposals of 32 points 217 -> 72 us, of 600 of 128 points 72 -> 41; with ping-pong
// buffers and 114 clusters resident they took 143 and 59).  At 512 points a CTA takes
// two butterflies per thread and stage: longer for one proposal, but without the
// clusters' idle half and waits more of them in a given time, so these take
// CTAs where more are listed than clusters fit (3000: 618 -> 495 us, 100: 34.8 ->
// 32.8; 60 stay at 24.6), unless they would come after larger ones on the same SMs (70 of
// 1024 points and 23 of 512: 44.7 us as clusters, 51.2 as CTAs; 53 and 40: 42.9 and 40.5) and are
// too few to make up for their length.  The sums keep the clusters' order: a partial one per
// channel and half of the bins, bins over lanes, lanes by halving distances, then
// warps in turn.
template <bool PERCH>
__global__ void __launch_bounds__(kHpThreads, 2) fd_hp_kernel(HpArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  grid_begin();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float2 red[32];
  __shared__ float4 s_part[2];  // this CTA's {rr hi, rr lo, hw hi, hw lo}, by turns
  __shared__ float4 s_small[4 * kHpSmallMax / 64];  // a small proposal's, per part and warp
  const int NFFT = a.NFFT;
  dc *S = reinterpret_cast<dc *>(smem_raw);
  const int r = (int)cluster.block_rank(), ch = r >> 1;
  const int ncl = (int)(gridDim.x >> 2);
  int cs[kNumBins];
  int total = 0;
#pragma unroll
  for (int b = kNumBins - 1; b >= 0; b--) {
    cs[b] = total;
    if ((32 << b) <= NFFT) total += a.bin_count[b];
  }
  if (total == 0) return;  // nothing listed: the counters are zero already
  // the bank's entries of bin q of channel c
  struct Bin {
    float4 gh, gl, wh, wl;
  };
  auto load_bin = [&](const HpEntry &e, int N, int c, int q, Bin &t) {
    const int j = e.imin + ((q + (N >> 1)) & (N - 1));  // fftshift
    if (j < 0 || j >= NFFT) return false;
    const size_t sj = (size_t)e.seg * NFFT + j;
    t = {a.g32[2 * sj + c], a.g32lo[2 * sj + c], a.w32[sj], a.w32lo[sj]};
    return true;
  };
  // residual and template power of a bin from the channel's two spectra there
  auto add_bin = [&](const HpEntry &e, const Bin &t, int c, dc s0, dc s1, df &rr, df &hw) {
    dc h = dc_add(dc_mul(s0, dc_from(make_float2(t.gh.x, t.gh.y), make_float2(t.gl.x, t.gl.y))),
                  dc_mul(s1, dc_from(make_float2(t.gh.z, t.gh.w), make_float2(t.gl.z, t.gl.w))));
    h = dc_scale2(h, e.amp_p2);
    const dc w = c == 0 ? dc_from(make_float2(t.wh.x, t.wh.y), make_float2(t.wl.x, t.wl.y))
                        : dc_from(make_float2(t.wh.z, t.wh.w), make_float2(t.wl.z, t.wl.w));
    rr = df_add(rr, df_sq_sum(dc_sub(w, h)));
    hw = df_add(hw, df_sq_sum(h));
  };
  // the large entries come first
  const int nlarge = cs[kHpSmallBins], n512 = cs[kHpSmallBins - 1] - nlarge;
  const bool cta512 = nlarge + n512 > ncl && (4 * nlarge + n512 <= 4 * ncl || nlarge + n512 > 4 * ncl);
  const int nbig = cta512 ? nlarge : nlarge + n512;
  int turn = 0;
  for (int k = (int)(blockIdx.x >> 2); k < nbig; k += ncl, turn ^= 1) {
    const HpEntry e = hp_entry(a, k, cs);
    const int N = e.N, ln = e.bin + 5;
    const float4 *src = a.series + e.off + (long long)r * N;
    for (int n0 = threadIdx.x; n0 < N; n0 += 4 * kHpThreads) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (n0 + u * kHpThreads < N) v[u] = src[n0 + u * kHpThreads];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (n0 + u * kHpThreads < N) S[hp_at(hp_rev(n0 + u * kHpThreads, ln))] = dc_from(v[u]);
    }
    // bins of this CTA's half
    const int half = N >> 1, q0 = (r & 1) * half;
    Bin t;
    bool has = (int)threadIdx.x < half && load_bin(e, N, ch, q0 + (int)threadIdx.x, t);
    __syncthreads();
    hp_fft(S, ln, 1, a.tw32x[e.bin]);
    cluster.sync();  // every spectrum of the proposal is complete
    const dc *Sp = cluster.map_shared_rank(S, (unsigned)(r ^ 1));
    const dc *S0 = (r & 1) ? Sp : S, *S1 = (r & 1) ? S : Sp;  // the channel's series 2c, 2c + 1
    df rr = {0.f, 0.f}, hw = {0.f, 0.f};
    for (int q = q0 + threadIdx.x; q < q0 + half; q += blockDim.x) {
      Bin next;
      const bool has_next = q + kHpThreads < q0 + half && load_bin(e, N, ch, q + kHpThreads, next);
      if (has) add_bin(e, t, ch, S0[hp_at(q)], S1[hp_at(q)], rr, hw);
      t = next;
      has = has_next;
    }
    rr = hp_block_sum(rr, red);
    hw = hp_block_sum(hw, red);
    if (threadIdx.x == 0) s_part[turn] = make_float4(rr.hi, rr.lo, hw.hi, hw.lo);
    cluster.sync();  // partial sums are published; the partner is done with S
    if (r == 0 && threadIdx.x == 0 && e.ok) {
      df s[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      for (int q = 0; q < 4; q++) {
        const float4 o = *cluster.map_shared_rank(&s_part[turn], (unsigned)q);
        s[q >> 1] = df_add(s[q >> 1], df{o.x, o.y});
        s[2] = df_add(s[2], df{o.z, o.w});
      }
      hp_write(e.item, N, e.seg, e.imin, NFFT, s, a.Q, a.QA, PERCH, a.term_x, a.dlogl, a.term_y, a.hh, a.term_ch,
               a.status);
    }
    // the next proposal's sums go to the other s_part, the one after it follows
    // two more cluster barriers
  }
  if ((int)(blockIdx.x >> 2) < nbig) cluster.sync();  // CTA 0 has read every s_part
  // small proposals, first on the CTAs that had no large one
  for (int k = nbig + (int)(gridDim.x - 1 - blockIdx.x); k < total; k += (int)gridDim.x) {
    const HpEntry e = hp_entry(a, k, cs);
    const int N = e.N, ln = e.bin + 5, half = N >> 1, tid = threadIdx.x;
    const float4 *src = a.series + e.off;
    for (int n = tid; n < 4 * N; n += kHpThreads)
      S[hp_at((n & ~(N - 1)) + hp_rev(n & (N - 1), ln))] = dc_from(src[n]);
    // part (channel, half of the bins) and bin of item i
    auto part = [&](int i) { return i >> (ln - 1); };
    auto bin = [&](int i) { return i & (N - 1); };
    Bin t;
    bool has = tid < 2 * N && load_bin(e, N, part(tid) >> 1, bin(tid), t);
    __syncthreads();
    hp_fft(S, ln, 4, a.tw32x[e.bin]);
    const int g = half < 32 ? half : 32;  // lanes of a part's partial sum
    for (int i = tid; i < 2 * N; i += kHpThreads) {  // whole warps
      Bin next;
      const bool has_next = i + kHpThreads < 2 * N && load_bin(e, N, part(i + kHpThreads) >> 1, bin(i + kHpThreads), next);
      const int c = part(i) >> 1, q = bin(i);
      df rr = {0.f, 0.f}, hw = {0.f, 0.f};
      if (has) add_bin(e, t, c, S[hp_at(2 * c * N + q)], S[hp_at((2 * c + 1) * N + q)], rr, hw);
      for (int off = g >> 1; off > 0; off >>= 1) {
        const df ro = {__shfl_xor_sync(0xffffffffu, rr.hi, off), __shfl_xor_sync(0xffffffffu, rr.lo, off)};
        const df ho = {__shfl_xor_sync(0xffffffffu, hw.hi, off), __shfl_xor_sync(0xffffffffu, hw.lo, off)};
        rr = df_add(rr, ro);
        hw = df_add(hw, ho);
      }
      if ((i & (g - 1)) == 0) s_small[i / g] = make_float4(rr.hi, rr.lo, hw.hi, hw.lo);
      t = next;
      has = has_next;
    }
    __syncthreads();  // the sums are published, and S is free
    if (tid == 0 && e.ok) {
      const int nw = half / g;
      df s[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      for (int p = 0; p < 4; p++) {
        df rr = {0.f, 0.f}, hw = {0.f, 0.f};
        for (int w = 0; w < nw; w++) {
          const float4 o = s_small[p * nw + w];
          rr = df_add(rr, df{o.x, o.y});
          hw = df_add(hw, df{o.z, o.w});
        }
        s[p >> 1] = df_add(s[p >> 1], rr);
        s[2] = df_add(s[2], hw);
      }
      hp_write(e.item, N, e.seg, e.imin, NFFT, s, a.Q, a.QA, PERCH, a.term_x, a.dlogl, a.term_y, a.hh, a.term_ch,
               a.status);
    }
  }
  // the last CTA leaves the counters it was given at zero
  __syncthreads();  // this one has read them
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(a.done, 1) == (int)gridDim.x - 1) {
      for (int q = 0; q < a.nzero; q++) a.zero_at[q] = 0;
      *a.done = 0;
    }
  }
}

static size_t hp_smem_bytes(int nmax) {
  return (size_t)(nmax > 4 * kHpSmallMax ? nmax : 4 * kHpSmallMax) * sizeof(dc);
}

template <bool PERCH>
static cudaError_t launch_hp(const HpArgs &a, int num_sms, cudaStream_t stream) {
  const size_t smem = hp_smem_bytes(a.nmax);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 4;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kHpThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_chained
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  static LaunchSetup setup[kNumBins];
  int ncl = 0;
  cudaError_t e = launch_setup(setup[fd_bin_of(a.nmax)], [&](int *o) {
    cudaError_t r = cudaFuncSetAttribute(fd_hp_kernel<PERCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)hp_smem_bytes(kMaxN));
    if (r != cudaSuccess) return r;
    cudaLaunchConfig_t q = cfg;
    q.gridDim = dim3(4 * num_sms);
    return cudaOccupancyMaxActiveClusters(o, fd_hp_kernel<PERCH>, &q);
  }, &ncl);
  if (e != cudaSuccess) return e;
  if (ncl < 1) ncl = 1;
  cfg.gridDim = dim3(4 * grid_for(ncl, a.nitems));
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, fd_hp_kernel<PERCH>, a);
}

// The double-float sine/cosine table of the current device, from
// extended-precision host values; once per device, when a context is created
// (a synchronous copy, never inside a stream capture).
cudaError_t fd_hp_tables_init() {
  static LaunchSetup setup;
  int done = 0;
  return launch_setup(setup, [&](int *o) {
    float4 t[64];
    for (int k = 0; k < 64; k++) {
      const long double x = (long double)k * (3.14159265358979323846264338327950288L / 32.0L);
      const long double sv = sinl(x), cv = cosl(x);
      const float sh = (float)sv, ch = (float)cv;
      t[k] = make_float4(sh, (float)(sv - (long double)sh), ch, (float)(cv - (long double)ch));
    }
    *o = 1;
    return cudaMemcpyToSymbol(g_hp_sincos, t, sizeof(t));
  }, &done);
}

cudaError_t fd_launch_reeval(const SlowArgs &sa, const HpArgs &h, bool perch, int num_sms, cudaStream_t stream,
                             int *nlaunch) {
  cudaError_t e;
  static LaunchSetup slow_setup;
  int occ = 0;
  e = launch_setup(slow_setup, [&](int *o) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, fd_slow_hp_kernel, 96, 0);
  }, &occ);
  if (e != cudaSuccess) return e;
  const int full = (occ > 0 ? occ : 1) * num_sms;
  e = launch_chained(fd_slow_hp_kernel, grid_for(full, sa.nitems * slow_chunks(sa.NFFT)), 96, 0, stream, sa);
  if (e != cudaSuccess) return e;
  e = perch ? launch_hp<true>(h, num_sms, stream) : launch_hp<false>(h, num_sms, stream);
  if (nlaunch) *nlaunch += 2;
  return e;
}

}  // namespace glass
