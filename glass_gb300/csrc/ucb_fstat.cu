// F-statistic of sky/frequency cells for sm_103a, FP64 (compiled without
// multiply-add contraction; multiply-adds are written out).
//
// The reference evaluates one cell at a time (get_Fstat_logL,
// ucb/src/glass_ucb_fstatistic.c:646-703): four filter waveforms by
// ucb_waveform (:231-348), their inner products with the data N^i (:350-409)
// and with each other M^ij (:411-516), M^-1 by LAPACK, logL = N^T M^-1 N / 2
// (:599-622) and the maximum-likelihood amplitude, inclination, polarisation
// and phase (:525-597, :624-644).  build_fstatistic_proposal
// (ucb/src/glass_ucb_proposal.c:1085-1182) calls it for every cell of a
// frequency x sky grid, with OpenMP over the sky rows.
//
// The four filters are two templates and their quarter turns.  At inclination
// pi/2 only the plus amplitude is left, so with H the response to e+ (psi = 0)
// and G the response to -ex (psi = pi/4, phase pi), the filters (psi, phase) =
// (0, 0), (pi/4, pi), (0, 3pi/2), (pi/4, pi/2) are H, G, iH, iG, exactly.  (The
// reference rounds each filter's carrier argument, ~1e6 rad, on its own, which
// moves its filters by ~1e-10 rad from these; the results agree to that.)  So
// N = (d.H, d.G, d.iH, d.iG) is two complex products, and of M only |H|^2,
// |G|^2 and the complex H*.G are left:
//   M = [ HH  Re  0  -Im ]     Re + i Im = sum H* G
//       [ Re  GG  Im  0  ]
//       [ 0   Im  HH  Re ]
//       [ -Im 0   Re  GG ]
//
// A batch of cells runs in four stages, the cells binned by their filter size
// N = ucb_bandwidth(f0, fdot, cos theta, A = 1e-22) in 16..4096:
//   plan    one thread per cell: the per-cell geometry;
//   slow    one thread per (cell, sample): the six arms' transfer factors
//           (slow_transfer64) once, with both real polarisation patterns;
//   spec    per size, one group of N/4 threads per cell: FFT of H's and G's
//           two series per channel, TDI weights and whitening per bin (the
//           likelihood path's tables), and the eight sums over the segment
//           bins 0 < k < NFFT;
//   finish  one thread per cell: the 4x4 solve, logL and the fit.
// All four are bound by the FP64 pipe (85% busy by ncu).  Against four filters,
// each with its own series, transforms and ten products, 1440 -> 314 FP64
// instructions per sample in the slow part and 656 -> 208 in the spectral part;
// the solve, one lane of a warp per cell before, runs full warps.  51200 cells
// of 64 samples: 13.43 -> 3.27 ms.
//
// The A/E inner products of the reference weight both channels with the A
// channel's noise C[0][0]; with templates and data whitened by their own
// channel's noise, the E terms are multiplied by invC_A/invC_E per bin, which
// gives the same weights.

#include "../../include/glass_gb300.h"
#include "ucb_fd.cuh"
#include "ucb_fd_device.cuh"

namespace glass {

namespace {

constexpr int kFsBins = 9;  // N = 16 << b
constexpr int kFsSeries = 8;  // (H, G) x (A2, A1, E2, E1)

struct FsCell {
  ItemF64 it;     // the cell's geometry, f0, fdot, q, amp/(2N), segment, N, imin
  // over the segment bins, whitened, before the amplitude: |H|^2, |G|^2, Re and
  // Im of H* G, Re and Im of d* H, Re and Im of d* G
  double sum[8];
  int live;       // evaluated (the others' results are written by the plan)
};

struct FsPlanArgs {
  int ncells, nseg, NFFT, cap;
  int seg_const;  // segment of every cell when cell_seg is null
  double T, fstar, L;
  const int *cell_seg;
  const double *cells;
  const int *seg_qmin;
  FsCell *fc;
  int *bin_count, *bin_list;
  double *logl, *fparams;
  int *status;
};

struct FsSlowArgs {
  int cap;
  const double2 *tw1024;
  const int *bin_count, *bin_list;
  const FsCell *fc;
  const OrbitSample64 *pos64[kNumBins];
  double2 *series;
};

struct FsSpecArgs {
  int NFFT, cap, bin;
  const int *bin_count, *bin_list;
  FsCell *fc;
  const double2 *series;
  const double2 *tw;  // twiddles of size N (size 16: every other entry of size 32's)
  int tw_stride;
  const double2 *w64, *g64;
  const double *rho;
};

// ------------------------------------------------------------ 4x4 algebra
// In-place inverse by Gauss-Jordan elimination with partial pivoting.
__device__ bool fs_invert4(double *m) {
  double a[4][8];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      a[i][j] = m[4 * i + j];
      a[i][4 + j] = (i == j) ? 1.0 : 0.0;
    }
  for (int c = 0; c < 4; c++) {
    int p = c;
    for (int r = c + 1; r < 4; r++)
      if (fabs(a[r][c]) > fabs(a[p][c])) p = r;
    if (a[p][c] == 0.0) return false;
    if (p != c)
      for (int j = 0; j < 8; j++) {
        double t = a[c][j];
        a[c][j] = a[p][j];
        a[p][j] = t;
      }
    const double inv = 1.0 / a[c][c];
    for (int j = 0; j < 8; j++) a[c][j] *= inv;
    for (int r = 0; r < 4; r++) {
      if (r == c) continue;
      const double f = a[r][c];
      if (f == 0.0) continue;
      for (int j = 0; j < 8; j++) a[r][j] -= f * a[c][j];
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) m[4 * i + j] = a[i][4 + j];
  return true;
}

// logL and the maximum-likelihood parameters from N (already times 4) and M
// (already times 4, full symmetric).  out: logL, A, iota, psi, phase.
// Returns false when M is singular but not zero.
__device__ bool fs_finish(const double *Nv, double *m, double *out) {
  // no filter bin inside the segment leaves M = 0, which LAPACK's
  // dgetrf/dgetri (utils/src/glass_math.c:501-523) leave as it is: logL = 0, a = 0
  bool any = false;
#pragma unroll
  for (int c = 0; c < 16; c++) any |= (m[c] != 0.0);
  if (any && !fs_invert4(m)) return false;
  // ucb/src/glass_ucb_fstatistic.c:612-621
  out[0] = 0.5 * (m[0] * Nv[0] * Nv[0] + 2 * m[1] * Nv[0] * Nv[1] + 2 * m[2] * Nv[0] * Nv[2] +
                  2 * m[3] * Nv[0] * Nv[3] + m[5] * Nv[1] * Nv[1] + 2 * m[6] * Nv[1] * Nv[2] +
                  2 * m[7] * Nv[1] * Nv[3] + m[10] * Nv[2] * Nv[2] + 2 * m[11] * Nv[2] * Nv[3] +
                  m[15] * Nv[3] * Nv[3]);
  // :636-643
  double a[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    a[i] = m[4 * i] * Nv[0] + m[4 * i + 1] * Nv[1] + m[4 * i + 2] * Nv[2] + m[4 * i + 3] * Nv[3];
  // :552-570
  const double a1p4 = a[0] + a[3], a2m3 = a[1] - a[2], a1m4 = a[0] - a[3], a2p3 = a[1] + a[2];
  const double Ap = sqrt(a1p4 * a1p4 + a2m3 * a2m3) + sqrt(a1m4 * a1m4 + a2p3 * a2p3);
  const double Ac = sqrt(a1p4 * a1p4 + a2m3 * a2m3) - sqrt(a1m4 * a1m4 + a2p3 * a2p3);
  double psi = atan2(Ap * a[3] - Ac * a[0], -(Ac * a[1] + Ap * a[2]));
  psi *= 0.5;
  const double sp = sin(2.0 * psi);
  const double c = (double)((sp > 0) - (sp < 0));
  out[1] = 0.5 * (Ap + sqrt(Ap * Ap - Ac * Ac));
  out[2] = acos(-Ac / (Ap + sqrt(Ap * Ap - Ac * Ac)));
  out[3] = psi;
  out[4] = atan2(c * (Ap * a[3] - Ac * a[0]), -c * (Ac * a[2] + Ap * a[1]));
  return true;
}

__device__ void fs_write(const FsPlanArgs &a, int i, const double *o, int st) {
  a.logl[i] = o[0];
  if (a.fparams)
#pragma unroll
    for (int k = 0; k < 4; k++) a.fparams[4 * (size_t)i + k] = o[1 + k];
  if (a.status) a.status[i] = st;
}

// ------------------------------------------------------------------- plan
// One thread per cell.  Filter parameters as get_filters sets them
// (ucb/src/glass_ucb_fstatistic.c:241-344): f0 T, cos theta, phi, ln 2,
// cos(pi/2), psi, phase (0, 0 for H), fdot T^2.
__global__ void __launch_bounds__(128) fs_plan_kernel(FsPlanArgs a) {
  grid_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int b = -1;
  if (i < a.ncells) {
    const double *x = a.cells + 4 * (size_t)i;
    const double f0 = x[0], fdot = x[1], theta = x[2], phi = x[3];
    const int seg = a.cell_seg ? a.cell_seg[i] : a.seg_const;
    const double nan = __longlong_as_double(0x7ff8000000000000ULL);
    double o[5] = {nan, nan, nan, nan, nan};
    if (seg < 0 || seg >= a.nseg) {
      fs_write(a, i, o, GLASS_ITEM_BAD_SEGMENT);
    } else if (!(isfinite(f0) && isfinite(fdot) && isfinite(theta) && isfinite(phi)) || !(f0 > 0.0)) {
      fs_write(a, i, o, GLASS_ITEM_NONFINITE);
    } else {
      const double costh = cos(theta);
      // the rule at amplitude 1e-22, in FP64 only where its FP32 interval leaves it
      // open (ln 1e-22 = -50.656872)
      const SpreadInterval sp = spread_interval(a.T, 1.0 / a.fstar, a.L, a.NFFT, f0, costh, -50.656872f,
                                                to_f32(fdot * (a.T * a.T)));
      const int N = sp.open() ? bandwidth_dev(a.L, a.fstar, f0, fdot, costh, 1.e-22, a.T, a.NFFT) : max(sp.D0, sp.S0);
      const long long q = (long long)(f0 * a.T);
      const long long qq = q - (long long)a.seg_qmin[seg];
      // filter bin i sits at segment bin qq + i - N/2 (:378, :423); bins
      // 0 < k < NFFT take part
      const long long lo = qq - N / 2, hi = lo + N - 1;
      if (N > kMaxN) {
        fs_write(a, i, o, GLASS_ITEM_NONFINITE);
      } else if (hi < 1 || lo >= a.NFFT) {
        double Nv[4] = {0, 0, 0, 0}, m[16] = {};
        fs_finish(Nv, m, o);
        fs_write(a, i, o, GLASS_ITEM_OUTSIDE);
      } else {
        ItemF64 c;
        double p[8];
        p[0] = f0 * a.T;
        p[1] = costh;
        p[2] = phi;
        p[3] = log(2.0);
        p[4] = cos(M_PI_2);
        p[5] = p[6] = 0.0;
        p[7] = fdot * (a.T * a.T);
        SourceGeom g;
        source_geometry(p, 8, a.T, g);
        make_item_f64(g, N, a.fstar, c);
        c.amp_s *= 0.5;  // the plus factor (1 + cos^2 iota) / 2, left out of H and G
        c.seg = seg;
        c.N = N;
        c.imin = (int)lo;
        a.fc[i].it = c;
        b = 31 - __clz(N) - 4;
      }
    }
  }
  if (i < a.ncells) a.fc[i].live = b >= 0;
  // warp-aggregated binning: one atomic per distinct size per warp
  const int lane = threadIdx.x & 31;
  const unsigned active = __ballot_sync(0xffffffffu, b >= 0);
  if (b >= 0) {
    const unsigned same = __match_any_sync(active, b);
    const int first = __ffs(same) - 1;
    int base = 0;
    if (lane == first) base = atomicAdd(&a.bin_count[b], __popc(same));
    base = __shfl_sync(same, base, first);
    a.bin_list[(size_t)b * a.cap + base + __popc(same & ((1u << lane) - 1))] = i;
  }
}

// Start (in samples of one series) of size bin `bin` in the scratch: sizes in
// increasing order, cells of one size back to back, 8 series of N each.
__device__ __forceinline__ long long fs_bin_start(const int *bin_count, int bin) {
  long long acc = 0;
#pragma unroll
  for (int b = 0; b < kFsBins; b++)
    if (b < bin) acc += (long long)bin_count[b] * (16 << b);
  return acc * kFsSeries;
}

// ------------------------------------------------------------------- slow
// One thread per (cell, sample): the six arm series of H and G (ucb/src/
// glass_ucb_waveform.c:840-922 with real polarisation factors), combined to the
// four A/E series each and stored at [cell][template][series][n].
__global__ void __launch_bounds__(256) fs_slow_kernel(FsSlowArgs a) {
  grid_begin();
  long long cs[kFsBins + 1];
  long long acc = 0;
#pragma unroll
  for (int b = 0; b < kFsBins; b++) {
    cs[b] = acc;
    acc += (long long)a.bin_count[b] << (b + 4);
  }
  cs[kFsBins] = acc;
  const long long total = acc;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < total; s += stride) {
    int b = 0;
#pragma unroll
    for (int bb = 1; bb < kFsBins; bb++)
      if (s >= cs[bb]) b = bb;
    const int N = 16 << b;
    const long long local = s - cs[b];
    const int slot = (int)(local >> (b + 4));
    const int n = (int)(local & (N - 1));
    const int cell = a.bin_list[(size_t)b * a.cap + slot];
    const ItemF64 &c = a.fc[cell].it;
    // size 16 samples are every other sample of size 32 (same times exactly)
    const OrbitSample64 &o = b == 0 ? a.pos64[0][2 * n] : a.pos64[b - 1][n];
    ArmGeom64 g;
    slow_geom64(c, o, g);
    constexpr int arm[6] = {0, 1, 0, 2, 1, 2};
    double2 w[6], d[6], cmb[4];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double arg2, h, aev;
      slow_sc64(c, o, i, arg2, h, aev);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int q = 2 * i + e;
        const bool back = i == 2 || (i == 1 && e == 0);
        const double2 t = slow_transfer64(h, back ? -g.kr[arm[q]] : g.kr[arm[q]], arg2, aev, a.tw1024);
        w[q] = make_double2(t.x, -t.y);
      }
    }
    double2 *out = a.series + fs_bin_start(a.bin_count, b) + (long long)slot * kFsSeries * N + n;
#pragma unroll
    for (int q = 0; q < 6; q++) d[q] = cscale(w[q], g.dp[arm[q]]);
    ae_combos64(d, cmb);
#pragma unroll
    for (int k = 0; k < 4; k++) out[(size_t)k * N] = cmb[k];
#pragma unroll
    for (int q = 0; q < 6; q++) d[q] = cscale(w[q], 2.0 * g.dc[arm[q]]);
    ae_combos64(d, cmb);
#pragma unroll
    for (int k = 0; k < 4; k++) out[(size_t)(4 + k) * N] = cmb[k];
  }
}

// ------------------------------------------------------------------- spec
template <int N>
struct FsCfg {
  static constexpr int GT = N / 4;
  static constexpr int CTA = GT >= 128 ? GT : 128;
  static constexpr int GPC = CTA / GT;
  static constexpr size_t smem = sizeof(double2) * (size_t)N * (1 + (size_t)GPC * 2) + sizeof(double) * 32 * GPC;
};

// One channel of one template at a time (two series in shared memory): H's bins
// stay in registers while G's series are transformed, then the channel's share
// of the eight sums is taken.
template <int N>
__global__ void __launch_bounds__(FsCfg<N>::CTA) fs_spec_kernel(FsSpecArgs a) {
  using Cfg = FsCfg<N>;
  constexpr int GT = Cfg::GT, GPC = Cfg::GPC;
  constexpr int B = N / GT;  // bins per thread (4)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grid_begin();
  const int count = a.bin_count[a.bin];
  if (count == 0) return;
  double2 *tw = reinterpret_cast<double2 *>(smem_raw);
  double2 *bufs = tw + N;
  double *reds = reinterpret_cast<double *>(bufs + (size_t)GPC * 2 * N);
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = a.tw[(size_t)i * a.tw_stride];
  __syncthreads();
  const double2 *ser_bin = a.series + fs_bin_start(a.bin_count, a.bin);
  const int *list = a.bin_list + (size_t)a.bin * a.cap;
  const int g = threadIdx.x / GT, lane = threadIdx.x % GT;
  double2 *buf = bufs + (size_t)g * 2 * N;
  double *red = reds + 32 * g;
  const int NFFT = a.NFFT;
  for (int base = blockIdx.x * GPC; base < count; base += gridDim.x * GPC) {
    const int slot = base + g;
    const bool valid = slot < count;
    if (base + (GT >= 32 ? g : (int)(threadIdx.x & ~31u) / GT) >= count) break;  // a warp with no cell
    const int sl = valid ? slot : count - 1;
    const int cell = list[sl];
    const ItemF64 &it = a.fc[cell].it;
    const int imin = it.imin;
    const size_t seg0 = (size_t)it.seg * NFFT;
    const double2 *ser = ser_bin + (size_t)sl * kFsSeries * N;
    double sum[8] = {};
#pragma unroll 1
    for (int chan = 0; chan < 2; ++chan) {
      double2 hb[B];
#pragma unroll 1
      for (int f = 0; f < 2; ++f) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int r = 0; r < B; ++r)
            buf[q * N + lane + GT * r] = ser[(size_t)(4 * f + 2 * chan + q) * N + lane + GT * r];
        group_bar<GT>(g);
        group_fft<N, GT, 2, 2>(buf, tw, lane, g);
#pragma unroll
        for (int r = 0; r < B; ++r) {
          const int k = lane + GT * r;
          const int j = imin + ((k + N / 2) & (N - 1));  // fftshift
          double2 h = make_double2(0.0, 0.0);
          if (j > 0 && j < NFFT) {
            const size_t sj = seg0 + j;
            const double2 g2 = a.g64[4 * sj + 2 * chan], g1 = a.g64[4 * sj + 2 * chan + 1];
            h = cfma(buf[k], g2, cmul(buf[N + k], g1));
            if (f == 1) {
              const double2 w = a.w64[2 * sj + chan];
              double2 H = hb[r], G = h;  // the second factors, weighted
              if (chan == 1) {
                const double rho = a.rho[sj];
                H = cscale(H, rho);
                G = cscale(G, rho);
              }
              sum[0] = fma(hb[r].x, H.x, fma(hb[r].y, H.y, sum[0]));
              sum[1] = fma(h.x, G.x, fma(h.y, G.y, sum[1]));
              sum[2] = fma(hb[r].x, G.x, fma(hb[r].y, G.y, sum[2]));
              sum[3] = fma(hb[r].x, G.y, fma(-hb[r].y, G.x, sum[3]));
              sum[4] = fma(w.x, H.x, fma(w.y, H.y, sum[4]));
              sum[5] = fma(w.x, H.y, fma(-w.y, H.x, sum[5]));
              sum[6] = fma(w.x, G.x, fma(w.y, G.y, sum[6]));
              sum[7] = fma(w.x, G.y, fma(-w.y, G.x, sum[7]));
            }
          }
          if (f == 0) hb[r] = h;
        }
        group_bar<GT>(g);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) sum[q] = group_sum<GT>(sum[q], red, lane, g);
    if (valid && lane == 0)
#pragma unroll
      for (int q = 0; q < 8; ++q) a.fc[cell].sum[q] = sum[q];
  }
}

// ----------------------------------------------------------------- finish
__global__ void __launch_bounds__(128) fs_finish_kernel(const FsCell *fc, int ncells, double *logl, double *fparams,
                                                        int *status) {
  grid_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncells || !fc[i].live) return;
  const double s = 4.0 * fc[i].it.amp_s, s2 = s * fc[i].it.amp_s;
  const double *v = fc[i].sum;
  const double Nv[4] = {s * v[4], s * v[6], -(s * v[5]), -(s * v[7])};
  const double hh = s2 * v[0], gg = s2 * v[1], re = s2 * v[2], im = s2 * v[3];
  double m[16] = {hh, re, 0.0, -im, re, gg, im, 0.0, 0.0, im, hh, re, -im, 0.0, re, gg};
  double o[5];
  int st = 0;
  if (!fs_finish(Nv, m, o)) {
    const double nan = __longlong_as_double(0x7ff8000000000000ULL);
    for (int q = 0; q < 5; q++) o[q] = nan;
    st = GLASS_ITEM_NONFINITE;
  } else if (!isfinite(o[0])) {
    st = GLASS_ITEM_NONFINITE;
  }
  logl[i] = o[0];
  if (fparams)
#pragma unroll
    for (int q = 0; q < 4; q++) fparams[4 * (size_t)i + q] = o[1 + q];
  if (status) status[i] = st;
}

template <int N>
cudaError_t fs_launch_spec(const FsSpecArgs &a, int ncells, int num_sms, cudaStream_t stream) {
  using Cfg = FsCfg<N>;
  static LaunchSetup setup;
  int occ = 0;
  cudaError_t e = launch_setup(setup, [&](int *o) {
    cudaError_t r = cudaFuncSetAttribute(fs_spec_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::smem);
    if (r != cudaSuccess) return r;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, fs_spec_kernel<N>, Cfg::CTA, Cfg::smem);
  }, &occ);
  if (e != cudaSuccess) return e;
  int need = (ncells + Cfg::GPC - 1) / Cfg::GPC;
  int grid = occ * num_sms;
  if (need < grid) grid = need;
  if (grid < 1) grid = 1;
  return launch_chained(fs_spec_kernel<N>, grid, Cfg::CTA, Cfg::smem, stream, a);
}


// ------------------------------------------------------- proposal grid
// Cell centres of the grid of build_fstatistic_proposal
// (ucb/src/glass_ucb_proposal.c:1119-1134), cell g = (i n_theta + j) n_phi + k.
__device__ __forceinline__ void fs_grid_centre(const FsGrid &G, int g, int &i, double &f, double &theta,
                                               double &phi) {
  i = g / (G.n_theta * G.n_phi);
  const int j = (g / G.n_phi) % G.n_theta, k = g % G.n_phi;
  f = G.fmin + i * G.d_f;
  f += G.d_f / 2;
  theta = acos((-1. + (double)j * G.d_theta + G.d_theta / 2));
  phi = (double)k * G.d_phi + G.d_phi / 2;
}

__global__ void fs_grid_cells_kernel(FsGrid G, int g0, int n, double *cells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i;
  double f, th, ph;
  fs_grid_centre(G, g0 + c, i, f, th, ph);
  double *x = cells + 4 * (size_t)c;
  x[0] = f;
  x[1] = 0.0;
  x[2] = th;
  x[3] = ph;
}

// Cells whose fdot = 0 value exceeds 1 get the chirp-mass scan (:1136-1148):
// their grid index goes to active[], their position in it to pos[].
__global__ void fs_scan_mark_kernel(const double *logl0, int n, int *count, int *active, int *pos) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  if (logl0[g] > 1) {
    const int idx = atomicAdd(count, 1);
    active[idx] = g;
    pos[g] = idx;
  } else {
    pos[g] = -1;
  }
}

__global__ void fs_scan_cells_kernel(FsGrid G, const int *active, int c0, int n, const double *fdot_tab,
                                     double *cells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const int a = (c0 + c) / kFsScan, s = (c0 + c) % kFsScan;
  int i;
  double f, th, ph;
  fs_grid_centre(G, active[a], i, f, th, ph);
  double *x = cells + 4 * (size_t)c;
  x[0] = f;
  x[1] = fdot_tab[(size_t)i * kFsScan + s];
  x[2] = th;
  x[3] = ph;
}

// logLmax over the fdot = 0 value and the scan up to its first value below 1,
// squared (:1138-1150).
__global__ void fs_finalize_kernel(const double *logl0, const int *pos, const double *scan, int n,
                                   double *tensor) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const double v0 = logl0[g];
  double mx = v0;
  if (v0 > 1) {
    const double *sv = scan + (size_t)pos[g] * kFsScan;
    for (int s = 0; s < kFsScan; s++) {
      const double v = sv[s];
      if (v > mx) mx = v;
      if (v < 1) break;
    }
  }
  tensor[g] = mx * mx;
}

}  // namespace

// ------------------------------------------------------------------- host
size_t fs_cell_bytes() { return sizeof(FsCell); }

// Largest filter size of a segment of NFFT bins: 2^floor(log2(NFFT/2)),
// at least 16 (ucb/src/glass_ucb_waveform.c:700-701).
int fs_max_size(int NFFT) {
  int half = NFFT / 2, n = 1;
  while (n * 2 <= half) n *= 2;
  return n < 16 ? 16 : n;
}

cudaError_t fs_work_alloc(FsWorkDev &w, int cap, int NFFT) {
  const int maxN = fs_max_size(NFFT) > kMaxN ? kMaxN : fs_max_size(NFFT);
  const size_t series = (size_t)cap * kFsSeries * maxN * sizeof(double2);
  if (w.mem && cap <= w.cap && series <= w.series_bytes) return cudaSuccess;
  cudaFree(w.mem);
  w = FsWorkDev{};
  size_t off_cells = 0;
  size_t off_count = (off_cells + sizeof(FsCell) * (size_t)cap + 255) / 256 * 256;
  size_t off_list = off_count + 256;
  size_t off_series = (off_list + sizeof(int) * kFsBins * (size_t)cap + 255) / 256 * 256;
  size_t total = off_series + series;
  cudaError_t e = cudaMalloc(&w.mem, total);
  if (e != cudaSuccess) {
    w.mem = nullptr;
    return e;
  }
  char *base = (char *)w.mem;
  w.cap = cap;
  w.cells = base + off_cells;
  w.bin_count = (int *)(base + off_count);
  w.bin_list = (int *)(base + off_list);
  w.series = base + off_series;
  w.series_bytes = series;
  return cudaSuccess;
}

void fs_work_free(FsWorkDev &w) {
  cudaFree(w.mem);
  w = FsWorkDev{};
}

cudaError_t fs_launch(const FdBankDev &bank, const FdTablesDev &tab, const double *rho, FsWorkDev &w, int ncells,
                      const int *cell_seg, int seg_const, const double *cells, double *logl, double *fparams,
                      int *status, int num_sms, cudaStream_t stream, int *nlaunch) {
  cudaError_t e;
  int launches = 0;
  const int maxN = fs_max_size(bank.NFFT);
  for (int off = 0; off < ncells; off += w.cap) {
    const int n = ncells - off < w.cap ? ncells - off : w.cap;
    if ((e = cudaMemsetAsync(w.bin_count, 0, sizeof(int) * 16, stream)) != cudaSuccess) return e;
    FsPlanArgs pa;
    pa.ncells = n;
    pa.nseg = bank.nseg;
    pa.NFFT = bank.NFFT;
    pa.cap = w.cap;
    pa.T = bank.T;
    pa.fstar = bank.fstar;
    pa.L = kLARM;
    pa.cell_seg = cell_seg ? cell_seg + off : nullptr;
    pa.seg_const = seg_const;
    pa.cells = cells + 4 * (size_t)off;
    pa.seg_qmin = bank.qmin;
    pa.fc = (FsCell *)w.cells;
    pa.bin_count = w.bin_count;
    pa.bin_list = w.bin_list;
    pa.logl = logl + off;
    pa.fparams = fparams ? fparams + 4 * (size_t)off : nullptr;
    pa.status = status ? status + off : nullptr;
    e = launch_chained(fs_plan_kernel, (n + 127) / 128, 128, 0, stream, pa);
    launches++;
    if (e != cudaSuccess) return e;

    FsSlowArgs sa;
    sa.cap = w.cap;
    sa.tw1024 = tab.tw64[fd_bin_of(kSincosTab)];
    sa.bin_count = w.bin_count;
    sa.bin_list = w.bin_list;
    sa.fc = (const FsCell *)w.cells;
    for (int b = 0; b < kNumBins; b++) sa.pos64[b] = tab.pos64[b];
    sa.series = (double2 *)w.series;
    {
      static LaunchSetup setup;
      int occ = 0;
      if ((e = launch_setup(setup, [&](int *o) {
             return cudaOccupancyMaxActiveBlocksPerMultiprocessor(o, fs_slow_kernel, 256, 0);
           }, &occ)) != cudaSuccess)
        return e;
      e = launch_chained(fs_slow_kernel, occ * num_sms, 256, 0, stream, sa);
      launches++;
      if (e != cudaSuccess) return e;
    }

    FsSpecArgs ca;
    ca.NFFT = bank.NFFT;
    ca.cap = w.cap;
    ca.bin_count = w.bin_count;
    ca.bin_list = w.bin_list;
    ca.fc = (FsCell *)w.cells;
    ca.series = (const double2 *)w.series;
    ca.w64 = bank.w64;
    ca.g64 = bank.g64;
    ca.rho = rho;
    for (int b = 0; b < kFsBins; b++) {
      const int N = 16 << b;
      if (N > maxN || N > kMaxN) break;
      ca.bin = b;
      ca.tw = b == 0 ? tab.tt64[0] : tab.tt64[b - 1];
      ca.tw_stride = b == 0 ? 2 : 1;
      switch (N) {
        case 16: e = fs_launch_spec<16>(ca, n, num_sms, stream); break;
        case 32: e = fs_launch_spec<32>(ca, n, num_sms, stream); break;
        case 64: e = fs_launch_spec<64>(ca, n, num_sms, stream); break;
        case 128: e = fs_launch_spec<128>(ca, n, num_sms, stream); break;
        case 256: e = fs_launch_spec<256>(ca, n, num_sms, stream); break;
        case 512: e = fs_launch_spec<512>(ca, n, num_sms, stream); break;
        case 1024: e = fs_launch_spec<1024>(ca, n, num_sms, stream); break;
        case 2048: e = fs_launch_spec<2048>(ca, n, num_sms, stream); break;
        default: e = fs_launch_spec<4096>(ca, n, num_sms, stream); break;
      }
      launches++;
      if (e != cudaSuccess) return e;
    }
    e = launch_chained(fs_finish_kernel, (n + 127) / 128, 128, 0, stream, (const FsCell *)w.cells, n, pa.logl,
                       pa.fparams, pa.status);
    launches++;
    if (e != cudaSuccess) return e;
  }
  if (nlaunch) *nlaunch = launches;
  return cudaSuccess;
}

cudaError_t fs_grid_cells(const FsGrid &G, int g0, int n, double *cells, cudaStream_t stream) {
  fs_grid_cells_kernel<<<(n + 255) / 256, 256, 0, stream>>>(G, g0, n, cells);
  return cudaGetLastError();
}

cudaError_t fs_scan_mark(const double *logl0, int n, int *count, int *active, int *pos, cudaStream_t stream) {
  fs_scan_mark_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logl0, n, count, active, pos);
  return cudaGetLastError();
}

cudaError_t fs_scan_cells(const FsGrid &G, const int *active, int c0, int n, const double *fdot_tab, double *cells,
                          cudaStream_t stream) {
  fs_scan_cells_kernel<<<(n + 255) / 256, 256, 0, stream>>>(G, active, c0, n, fdot_tab, cells);
  return cudaGetLastError();
}

cudaError_t fs_finalize(const double *logl0, const int *pos, const double *scan, int n, double *tensor,
                        cudaStream_t stream) {
  fs_finalize_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logl0, pos, scan, n, tensor);
  return cudaGetLastError();
}

}  // namespace glass
