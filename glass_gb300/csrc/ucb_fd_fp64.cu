// Instantiations of the slow-part and per-size spectral kernels, plain FP64.
#include <cooperative_groups.h>

#include "ucb_fd_device.cuh"

namespace glass {

cudaError_t fd_launch_slow_fp64(const SlowArgs &a, int num_sms, cudaStream_t stream) {
  return launch_slow<false>(a, num_sms, stream);
}


cudaError_t fd_launch_spec_fp64(int N, const SpecArgs &a, int nitems, int num_sms, cudaStream_t stream,
                                bool perch) {
  if (perch) {
    switch (N) {
      case 2048: return launch_spec<2048, false, true>(a, nitems, num_sms, stream);
      case 4096: return launch_spec<4096, false, true>(a, nitems, num_sms, stream);
    }
    return cudaErrorInvalidValue;
  }
  switch (N) {
    case 32: return launch_spec<32, false>(a, nitems, num_sms, stream);
    case 64: return launch_spec<64, false>(a, nitems, num_sms, stream);
    case 128: return launch_spec<128, false>(a, nitems, num_sms, stream);
    case 256: return launch_spec<256, false>(a, nitems, num_sms, stream);
    case 512: return launch_spec<512, false>(a, nitems, num_sms, stream);
    case 1024: return launch_spec<1024, false>(a, nitems, num_sms, stream);
    case 2048: return launch_spec<2048, false>(a, nitems, num_sms, stream);
    case 4096: return launch_spec<4096, false>(a, nitems, num_sms, stream);
  }
  return cudaErrorInvalidValue;
}

cudaError_t fd_launch_spec_all_fp64(const SpecAllArgs &A, int num_sms, cudaStream_t stream, bool perch) {
  if (perch) return launch_spec_all<false, true>(A, num_sms, stream);
  return launch_spec_all<false>(A, num_sms, stream);
}

// A cluster of four CTAs per proposal, every size, for batches of at most a fifth as
// many proposals as SMs: CTA r transforms series r, and then sums half of its
// channel's bins from its own spectrum and its partner's (through distributed shared
// memory), so that a proposal's FP64 instructions run on four SMs; and the 2048- and
// 4096-point sizes need no launches of their own.  A host call of one proposal of 128
// points 31.0 -> 29.8 us, of 1024 66.9 -> 37.0, of 4096 207 -> 73; of 30 proposals of
// 512 points 53.4 -> 39.5, of 64 points 30.9 -> 31.0.  With more proposals than that the
// clusters queue and small sizes lose: of 76 of 128 points 34.8 -> 35.9.
template <bool PERCH>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(kSpecAllThreads) fd_spec_cluster64_kernel(SpecSmallArgs A) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  grid_begin();
  const SpecArgs &a = A.a;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[64];
  __shared__ double2 s_sum;
  const int r = (int)cluster.block_rank(), ch = r >> 1, tid = threadIdx.x, NFFT = a.NFFT;
  // this cluster's proposal: the k-th over the size lists
  int sl = (int)(blockIdx.x >> 2), b = 0;
  for (; b < A.nbins && sl >= a.bin_count[b]; b++) sl -= a.bin_count[b];
  if (b < A.nbins) {
    const int ln = b + 5, N = 32 << b;
    double2 *S = reinterpret_cast<double2 *>(smem_raw), *tw = S + N;
    const bool lok = chk(sl >= 0 && sl < a.cap, kChkBinList);
    const int item = lok ? a.bin_list[(size_t)b * a.cap + sl] : 0;
    const bool iok = chk(item >= 0 && item < a.nitems, kChkItem);
    int seg = 0, imin = 0;
    double s = 0.0;
    if (iok) {
      seg = a.items64[item].seg;
      imin = a.items64[item].imin;
      s = a.items64[item].amp_s;
    }
    const long long s0 = (bin_sample_start(a.bin_count, NFFT, b) + (long long)sl * N) * 4;
    const bool sok = chk(seg >= 0 && seg < a.nseg, kChkBankRead);
    const bool rok = chk(s0 + 4LL * N <= a.series_len, kChkSeriesRead);
    const bool inb = lok && iok && sok && rok;
    if (!inb) seg = 0;
    const double2 *src = reinterpret_cast<const double2 *>(a.series) + (inb ? s0 + (long long)r * N : 0);
    for (int i = tid; i < N; i += kSpecAllThreads) {
      S[hp_rev(i, ln)] = src[i];
      tw[i] = A.tw[b][i];
    }
    __syncthreads();
    fft4_dit64<1>(S, ln, tw);
    cluster.sync();  // every spectrum is complete
    const double2 *P0 = cluster.map_shared_rank(S, (unsigned)(2 * ch));
    const double2 *P1 = cluster.map_shared_rank(S, (unsigned)(2 * ch + 1));
    double wv = 0.0, hv = 0.0;
    for (int k = (r & 1) * (N / 2) + tid; k < ((r & 1) + 1) * (N / 2); k += kSpecAllThreads) {
      const int j = imin + ((k + N / 2) & (N - 1));  // fftshift
      if (j < 0 || j >= NFFT) continue;
      const size_t sj = (size_t)seg * NFFT + j;
      const double2 w = a.w64[2 * sj + ch];
      const double2 g2 = a.g64[4 * sj + 2 * ch], g1 = a.g64[4 * sj + 2 * ch + 1];
      const double2 h = cfma(P0[k], g2, cmul(P1[k], g1));
      wv = fma(w.x, h.x, fma(w.y, h.y, wv));
      hv = fma(h.x, h.x, fma(h.y, h.y, hv));
    }
    wv = group_sum<kSpecAllThreads>(wv, red, tid, 0);
    hv = group_sum<kSpecAllThreads>(hv, red + 32, tid, 0);
    if (tid == 0) s_sum = make_double2(wv, hv);
    cluster.sync();  // the sums are published
    if (r == 0 && tid == 0 && inb) {
      double2 q[4];
      for (int m = 0; m < 4; m++) q[m] = *cluster.map_shared_rank(&s_sum, (unsigned)m);
      double wA = q[0].x + q[1].x, hA = q[0].y + q[1].y, wE = q[2].x + q[3].x, hE = q[2].y + q[3].y;
      // 2 (w|h) - |h|^2 with the amplitude s
      double term;
      if (PERCH) {
        const double tA = s * (2.0 * wA - s * hA), tE = s * (2.0 * wE - s * hE);
        a.term_ch[2 * (size_t)item] = tA;
        a.term_ch[2 * (size_t)item + 1] = tE;
        term = tA + tE;
      } else {
        term = s * (2.0 * (wA + wE) - s * (hA + hE));
      }
      const double tx = a.term_x ? a.term_x[item] : 0.0;
      a.dlogl[item] = term - tx;
      if (a.term_y) a.term_y[item] = term;
      if (a.hh) a.hh[item] = 2.0 * (s * s) * (hA + hE);
      if (a.status) a.status[item] = isfinite(term) ? 0 : 1;
    }
    cluster.sync();  // no CTA leaves while CTA 0 may be reading its sum
  }
  // the last CTA leaves the size counts at zero
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(A.done, 1) == (int)gridDim.x - 1) {
      for (int q = 0; q < kNumBins; q++) A.zero_counts[q] = 0;
      *A.done = 0;
    }
  }
}

template <bool PERCH>
static cudaError_t launch_spec_cluster64(const SpecSmallArgs &A, cudaStream_t stream) {
  const size_t most = 2 * (size_t)kMaxN * sizeof(double2);
  static LaunchSetup setup;
  int done = 0;
  const cudaError_t e = launch_setup(setup, [&](int *o) {
    *o = 1;
    return cudaFuncSetAttribute(fd_spec_cluster64_kernel<PERCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  }, &done);
  if (e != cudaSuccess) return e;
  const size_t smem = 2 * ((size_t)32 << (A.nbins - 1)) * sizeof(double2);
  return launch_chained(fd_spec_cluster64_kernel<PERCH>, 4 * A.a.nitems, kSpecAllThreads, smem, stream, A);
}
cudaError_t fd_launch_spec_cluster_fp64(const SpecSmallArgs &A, cudaStream_t stream, bool perch) {
  return perch ? launch_spec_cluster64<true>(A, stream) : launch_spec_cluster64<false>(A, stream);
}

}  // namespace glass
