// Launches of the window correlation: the dispatch to the fused kernels (one
// translation unit per FFT size, k_corr_<N>.cu), the general-shape kernel,
// the analysis of caller-supplied planes and the peak epilogue.
#include "hh_attr.h"
#include "hh_corr_peaks.cuh"

namespace hh {

// the general-shape kernel (any FFT lengths, rectangular windows, planes
// larger than a CTA's shared memory)
#include "hh_corr_general.cuh"
// ... and the same with the plane in shared memory
#include "hh_corr_plane.cuh"

// Device analysis of caller-supplied planes (one CTA of 128 threads each).
// The plane is staged in shared memory when it fits (lds, the stride of its
// columns there), else read in place from global memory (lds = 0: planes above
// 200 KB, 256 x 256 and larger). The scan's threads walk neighbouring columns,
// so the stride is odd: with one of 32, 64 or 128 floats a warp's 32 columns
// meet in one bank (0.29 ms for 961 planes of 128 x 128 against 0.09, 0.32
// ms for 16129 of 32 x 32 against 0.17). The copy runs through the plane in
// order, all threads at work whatever its rows, and 64 registers leave 8 CTAs
// per SM: 10000 planes of 16 x 16 103 -> 83 us, of 32 x 32 122 -> 106 against a
// lane per row and 72 registers.
__global__ void __launch_bounds__(128, 8) analyze_planes_kernel(const AnalyzeArgs a, int lds) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int64_t P = (int64_t)a.nr * a.nc;
  float* R = reinterpret_cast<float*>(smem_raw);
  uint32_t* red = reinterpret_cast<uint32_t*>(smem_raw + (size_t)lds * a.nc * sizeof(float));
  float* s_vals = reinterpret_cast<float*>(red + 8 * KMAX);
  int* s_locs = reinterpret_cast<int*>(s_vals + KMAX);
  const int K = a.npeaks > 2 ? a.npeaks : 2;
  PeakOut po{a.du, a.dv, a.ratio, a.moment, a.alt_u, a.alt_v, a.nalt, a.G, a.packed, a.locs};
  const ScanPlan sp = scan_plan(threadIdx.x, 128, 0, a.nr - 1, 0, a.nc - 1);
  const int er = threadIdx.x % a.nr, ec = threadIdx.x / a.nr, sr = 128 % a.nr, sc = 128 / a.nr;
  for (int64_t pl = blockIdx.x; pl < a.nplanes; pl += gridDim.x) {
    const float* Rp = a.planes + pl * P;
    if (lds) {
      // element e of the plane at (e % nr, e / nr), by running indices
      int r = er, c = ec;
#pragma unroll 8
      for (int e = threadIdx.x; e < P; e += 128) {
        R[c * lds + r] = __ldg(Rp + e);
        r += sr;
        c += sc;
        if (r >= a.nr) {
          r -= a.nr;
          ++c;
        }
      }
      Rp = R;
    }
    __syncthreads();
    const int64_t gid = a.jobs ? (int64_t)a.jobs[4 * pl] + (int64_t)a.jobs[4 * pl + 1] * a.ny : -1;
    analyze_group(Rp, a.nr, a.nc, lds ? lds : a.nr, K, a.npeaks, a.finder, a.subpixel, threadIdx.x, 128, red, true, s_vals,
                  s_locs, gid, pl, &po, false, 0, sp, nullptr, 0);
    __syncthreads();
  }
}

// The per-window outputs from the peak records: the same arithmetic as the
// in-kernel epilogue, a thread per window, or while the windows are few
// (EPI_SPLIT) a thread per window and peak (blockIdx.y), so that the FP64
// logarithms of a window's peaks do not wait for one another. One thread / one
// per peak: 225 windows 10.5 / 6.4 us, 16129 windows 12 / 9 us (latency); 1.0 M
// windows a third longer when split (every thread reads the values again).
constexpr int64_t EPI_SPLIT = 32768;
template <bool SPLIT> __global__ void __launch_bounds__(128) peak_epilogue_kernel(const CorrArgs a, int N) {
  const int K = a.npeaks > 2 ? a.npeaks : 2;
  const int m0 = SPLIT ? blockIdx.y : 0, m1 = SPLIT ? m0 + 1 : K;
  const int64_t S = a.njobs;
  const PeakOut po{a.du, a.dv, a.ratio, a.moment, a.alt_u, a.alt_v, a.nalt, a.G, a.packed, a.locs};
  for (int64_t job = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; job < a.njobs;
       job += (int64_t)gridDim.x * blockDim.x) {
    const int nf = __float_as_int(__ldg(a.rec + job));
    if (nf < 0) continue;  // skipped by the correlation kernel
    int64_t gid;
    PeakOut pw = po;
    if (a.bp) {  // the correlation kernel's addressing of the window's grid cell
      const int p = a.jobs[4 * job];
      const BPair& b = a.bp[p];
      const int gij = a.jobs[4 * job + 1];
      gid = b.goff + (int64_t)(gij & 0xFFFF) + (int64_t)(gij >> 16) * b.ny;
      pw.G = (int64_t)b.ny * b.nx;
      pw.nalt = b.nalt;
      pw.alt_u = a.alt_u ? a.alt_u + b.aoff - b.goff : nullptr;
      pw.alt_v = a.alt_v ? a.alt_v + b.aoff - b.goff : nullptr;
    } else {
      gid = (int64_t)a.jobs[4 * job] + (int64_t)a.jobs[4 * job + 1] * a.ny;
    }
    float vals[KMAX];
    int locs[2 * KMAX];
    for (int m = 0; m < nf; ++m) {
      vals[m] = __ldg(a.rec + (int64_t)(1 + m) * S + job);
      if (SPLIT && m != m0) continue;
      locs[2 * m] = __float_as_int(__ldg(a.rec + (int64_t)(1 + K + 2 * m) * S + job));
      locs[2 * m + 1] = __float_as_int(__ldg(a.rec + (int64_t)(2 + K + 2 * m) * S + job));
    }
    peak_outputs(RecSrc{a.rec + job, S, K}, N, N, K, a.npeaks, a.subpixel, nf, vals, locs, gid, job, pw, m0, m1);
  }
}

cudaError_t launch_peak_epilogue(const CorrArgs& a, int N, cudaStream_t s, int num_sms) {
  int64_t eb = (a.njobs + 127) / 128;
  if (eb > (int64_t)num_sms * 16) eb = (int64_t)num_sms * 16;
  // the peaks past npeaks have no outputs but their packed words and locations
  const int K = a.npeaks > 2 ? a.npeaks : 2, peaks = a.packed || a.locs ? K : (a.npeaks > 1 ? a.npeaks : 1);
  if (a.njobs <= EPI_SPLIT) peak_epilogue_kernel<true><<<dim3((unsigned)eb, (unsigned)peaks), 128, 0, s>>>(a, N);
  else peak_epilogue_kernel<false><<<(unsigned)eb, 128, 0, s>>>(a, N);
  return cudaGetLastError();
}

size_t gcorr_plane_smem(int nr, int nc, int box_rows, int box_cols, int threads) {
  return plane_smem(nr, nc, box_rows, box_cols, threads / 32);
}

size_t correlate_record_words(int npeaks) { return (size_t)rec_words(npeaks > 2 ? npeaks : 2); }

#define HH_CORR_SIZES(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128)
#define X(n) cudaError_t launch_corr_##n(const CorrArgs& a, int W, cudaStream_t s, int num_sms);
HH_CORR_SIZES(X)
#undef X

bool correlate_supported(int N, int W) {
#define X(n) if (N == n && (W == n || 2 * W == n)) return true;
  HH_CORR_SIZES(X)
#undef X
  return false;
}

cudaError_t launch_correlate(const CorrArgs& a, int N, int W, cudaStream_t s, int num_sms) {
  if (a.njobs <= 0) return cudaSuccess;
#define X(n) if (N == n && (W == n || 2 * W == n)) return launch_corr_##n(a, W, s, num_sms);
  HH_CORR_SIZES(X)
#undef X
  return cudaErrorInvalidValue;
}

int gcorr_radix_plan(int n, int8_t* radix) {
  if (n < 1) return -1;
  int ns = 0;
  auto push = [&](int r) {
    if (ns >= 24) return false;
    radix[ns++] = (int8_t)r;
    return true;
  };
  while (n % 4 == 0) {
    if (!push(4)) return -1;
    n /= 4;
  }
  while (n % 2 == 0) {
    if (!push(2)) return -1;
    n /= 2;
  }
  for (int f = 3; f <= 61 && n > 1; f += 2)
    while (n % f == 0) {
      if (!push(f)) return -1;
      n /= f;
    }
  return n == 1 ? ns : -1;
}

cudaError_t launch_correlate_general(const CorrArgs& a, cudaStream_t s) {
  if (a.njobs <= 0) return cudaSuccess;
  if (!a.twr || !a.twc || a.gscr_slices < 1 || a.gc_smem_bytes > 227 * 1024) return cudaErrorInvalidValue;
  if (!a.gc_in_smem && (!a.gscr || a.gc_col_warps < 1 || a.gc_col_warps > a.gc_threads / 32 || a.gc_chunk_c < 2))
    return cudaErrorInvalidValue;
  const bool boxed = a.gc_box[0] > 0 || a.gc_box[2] > 0 || a.gc_box[1] < a.nfr - 1 || a.gc_box[3] < a.nfc - 1;
  // a box smaller than the plane leaves its last row and column out
  if (boxed && (a.gc_box[1] > a.nfr - 2 || a.gc_box[3] > a.nfc - 2)) return cudaErrorInvalidValue;
  if (a.gc_in_smem) switch (a.gc_threads) {
      case 128: return boxed ? launch_plane<128, true>(a, s) : launch_plane<128, false>(a, s);
      case 256: return boxed ? launch_plane<256, true>(a, s) : launch_plane<256, false>(a, s);
      case 512: return boxed ? launch_plane<512, true>(a, s) : launch_plane<512, false>(a, s);
    }
  else switch (a.gc_threads) {
      case 256: return boxed ? launch_general<256, true>(a, s) : launch_general<256, false>(a, s);
      case 512: return boxed ? launch_general<512, true>(a, s) : launch_general<512, false>(a, s);
    }
  return cudaErrorInvalidValue;
}

cudaError_t launch_analyze_planes(const AnalyzeArgs& a, cudaStream_t s) {
  if (a.nplanes <= 0) return cudaSuccess;
  const size_t extra = 8 * KMAX * sizeof(uint32_t) + KMAX * sizeof(float) + 2 * KMAX * sizeof(int) + 16;
  int lds = a.nr | 1;
  if ((size_t)lds * a.nc * sizeof(float) + extra > 200 * 1024) lds = a.nr;
  if ((size_t)lds * a.nc * sizeof(float) + extra > 200 * 1024) lds = 0;
  const size_t sm = (size_t)lds * a.nc * sizeof(float) + extra;
  cudaError_t e = cudaFuncSetAttribute(analyze_planes_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return e;
  int64_t grid = a.nplanes < 4096 ? a.nplanes : 4096;
  analyze_planes_kernel<<<(unsigned)grid, 128, sm, s>>>(a, lds);
  return cudaGetLastError();
}

}  // namespace hh
