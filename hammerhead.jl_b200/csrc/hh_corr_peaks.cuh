// Peak analysis and spectrum helpers shared by the correlation kernels (the
// fused ones of hh_corr_fused.cuh, the general-shape one and the plane
// analysis of k_correlate.cu).
#pragma once
#include <math.h>
#include <stdint.h>

#include "hh_batch.h"
#include "hh_fft.cuh"
#include "hh_internal.h"

namespace hh {

// ---------------------------------------------------------------------------
// Global loads with L1 eviction hints. The shared-memory carveout leaves a
// small L1, and the window pixels, read once per window, would otherwise
// push out the small per-class tables (apodization, overlap gain, phase
// filter) that every window reads: the pixels stream past L1, the tables
// are kept. Inputs are read-only for the kernel's lifetime (.nc).
__device__ __forceinline__ float ld_stream(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint8_t ld_stream(const uint8_t* p) {
  unsigned short v;
  asm("ld.global.nc.L1::no_allocate.u8 %0, [%1];" : "=h"(v) : "l"(p));
  return (uint8_t)v;
}
// the same where `on`, else 0, as one predicated load: a branch per pixel
// would send the loads of a window out one by one
__device__ __forceinline__ float ld_stream_if(const float* p, bool on) {
  float v;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.nc.L1::no_allocate.f32 %0, [%1];\n\t}"
      : "=f"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ uint8_t ld_stream_if(const uint8_t* p, bool on) {
  unsigned short v;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.u16 %0, 0;\n\t"
      "@p ld.global.nc.L1::no_allocate.u8 %0, [%1];\n\t}"
      : "=h"(v) : "l"(p), "r"((int)on));
  return (uint8_t)v;
}
__device__ __forceinline__ float ld_keep_if(const float* p, bool on) {
  float v;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.nc.f32 %0, [%1];\n\t}"
      : "=f"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float ld_keep(const float* p) {
  float v;
  asm("ld.global.nc.L1::evict_last.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// Peak keys: larger key = larger value, ties broken by smaller column-major
// index (the reference's first-in-scan-order rule).
__device__ __forceinline__ uint32_t fkey(float v) {
  v = v + 0.0f;  // -0 -> +0 (they compare equal in the reference)
  uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Per-thread list of the best keys seen, descending, in KC register slots
// (KC >= K: 4 when the pass keeps at most 4 peaks, else KMAX).
template <int KC> struct TopK {
  uint32_t hi[KC];
  uint32_t lo[KC];
  int cnt;
  uint32_t thr;  // key of the K-th entry once the list is full, else 0
  __device__ __forceinline__ void init() {
    cnt = 0;
    thr = 0u;
#pragma unroll
    for (int m = 0; m < KC; ++m) hi[m] = lo[m] = 0u;
  }
  // the K-th (last retained) key, read with unrolled selects so the arrays
  // stay in registers for a run-time K
  __device__ __forceinline__ uint32_t last_hi(int K) const {
    uint32_t v = 0u;
#pragma unroll
    for (int m = 0; m < KC; ++m) v = (m == K - 1) ? hi[m] : v;
    return v;
  }
  __device__ __forceinline__ uint32_t last_lo(int K) const {
    uint32_t v = 0u;
#pragma unroll
    for (int m = 0; m < KC; ++m) v = (m == K - 1) ? lo[m] : v;
    return v;
  }
  // insert keeping (hi, lo) descending; K <= KC entries retained. Valid keys
  // are nonzero and empty slots hold 0, so the slots the new key beats are a
  // suffix of the first K: the first of them takes the new key, the others
  // their predecessor, and a key that beats none changes nothing. The
  // comparisons are independent of one another (no data-dependent indexing:
  // the list stays in registers).
  __device__ __forceinline__ void insert(uint32_t h, uint32_t l, int K) {
    bool b[KC];
#pragma unroll
    for (int m = 0; m < KC; ++m) b[m] = m < K && (h > hi[m] || (h == hi[m] && l > lo[m]));
#pragma unroll
    for (int m = KC - 1; m >= 0; --m) {
      const int q = m > 0 ? m - 1 : 0;
      const bool prev = m > 0 && b[q];
      const uint32_t ph = prev ? hi[q] : h, pl = prev ? lo[q] : l;
      hi[m] = b[m] ? ph : hi[m];
      lo[m] = b[m] ? pl : lo[m];
    }
    if (cnt < K) ++cnt;
    if (cnt == K) thr = last_hi(K);
  }
  __device__ __forceinline__ void pop() {
#pragma unroll
    for (int m = 0; m + 1 < KC; ++m) {
      hi[m] = hi[m + 1];
      lo[m] = lo[m + 1];
    }
    hi[KC - 1] = lo[KC - 1] = 0u;
    if (cnt > 0) --cnt;
    thr = 0u;
  }
};

// is_local_maximum (src/localmax.jl:3-19) on a column-major plane with
// leading dimension ldr: earlier neighbours (column-major) must be <=,
// later ones must be <; NaN is never a maximum.
__device__ __forceinline__ bool is_local_max(const float* R, int nr, int nc, int ldr, int r, int c, float I0) {
  if (isnan(I0)) return false;
  const int r0 = r > 0 ? r - 1 : 0, r1 = r < nr - 1 ? r + 1 : nr - 1;
  const int c0 = c > 0 ? c - 1 : 0, c1 = c < nc - 1 ? c + 1 : nc - 1;
  for (int jj = c0; jj <= c1; ++jj)
    for (int ii = r0; ii <= r1; ++ii) {
      if (ii == r && jj == c) continue;
      float In = R[jj * ldr + ii];
      bool earlier = (jj < c) || (jj == c && ii < r);
      if (earlier ? (In > I0) : (In >= I0)) return false;
    }
  return true;
}

// Lanes of the calling thread's group within its warp: the whole warp for
// groups of 32 threads or more, else the aligned block of `count` lanes
// (count a power of two below 32: two or more groups share a warp).
__device__ __forceinline__ unsigned grp_mask(int count) {
  return count >= 32 ? 0xffffffffu : (((1u << count) - 1u) << ((threadIdx.x & 31) & ~(count - 1)));
}

// Barrier of one thread group: lanes of a warp (count <= 32), the whole CTA
// (bar 0), or the named barrier `bar` shared by `count` threads (whole warps).
__device__ __forceinline__ void grp_sync(int bar, int count) {
  if (count <= 32) __syncwarp(grp_mask(count));
  else if (bar == 0) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(count) : "memory");
}

// Group-wide argmax of (hi, lo) keys. Every thread of the group calls it (it
// synchronises the group); each group has its own reduction slots.
__device__ __forceinline__ void group_argmax(uint32_t hi, uint32_t lo, uint32_t* red, int gwarp, int gsize,
                                             uint32_t& whi, uint32_t& wlo, int bar) {
  const int lane = threadIdx.x & 31, nwarps = gsize >> 5;
  const unsigned m = grp_mask(gsize);
  uint32_t mhi = __reduce_max_sync(m, hi);
  uint32_t mlo = __reduce_max_sync(m, hi == mhi ? lo : 0u);
  if (nwarps <= 1) {  // one warp or part of one: the shuffle reduction is the answer
    whi = mhi;
    wlo = mlo;
    return;
  }
  if (lane == 0) {
    red[2 * gwarp] = mhi;
    red[2 * gwarp + 1] = mlo;
  }
  grp_sync(bar, nwarps * 32);
  whi = 0u;
  wlo = 0u;
  for (int w = 0; w < nwarps; ++w) {
    uint32_t h = red[2 * w], l = red[2 * w + 1];
    if (h > whi || (h == whi && l > wlo)) {
      whi = h;
      wlo = l;
    }
  }
  grp_sync(bar, nwarps * 32);
}

// The K best keys over the lists of the lanes in `mask` (a warp or the
// group's part of one), by K shuffle rounds (keys are unique, so exactly one
// lane pops each winner): lane m receives the m-th best in (mh, ml);
// returns how many exist (the same in every lane).
template <class TK>
__device__ __forceinline__ int warp_topk(TK& tk, int K, int lane, uint32_t& mh, uint32_t& ml, unsigned mask) {
  int n = 0;
  mh = ml = 0u;
  for (int round = 0; round < K; ++round) {
    const uint32_t h = tk.hi[0], l = tk.lo[0];  // empty slots hold 0
    const uint32_t wh = __reduce_max_sync(mask, h);
    if (wh == 0u) break;
    const uint32_t wl = __reduce_max_sync(mask, h == wh ? l : 0u);
    if (h == wh && l == wl) tk.pop();
    if (lane == round) {
      mh = wh;
      ml = wl;
    }
    n = round + 1;
  }
  return n;
}

// Plane access for the subpixel and moment arithmetic: value at (row i,
// column j), 0-based. PlaneAcc reads a column-major plane with leading
// dimension ld; RecAcc reads a w x w patch around a peak kept in a peak
// record (column-major, `stride` words between consecutive cells).
struct PlaneAcc {
  const float* p;
  int ld;
  __device__ __forceinline__ float operator()(int i, int j) const { return p[j * ld + i]; }
};
// a plane that is zero, and not stored, outside rows [rlo, rhi] x columns [clo, chi]
struct BoxAcc {
  const float* p;
  int ld, rlo, rhi, clo, chi;
  __device__ __forceinline__ float operator()(int i, int j) const {
    return i >= rlo && i <= rhi && j >= clo && j <= chi ? p[j * ld + i] : 0.f;
  }
};
struct RecAcc {
  const float* p;
  int64_t stride;
  int i0, j0, w;  // patch origin and size
  __device__ __forceinline__ float operator()(int i, int j) const {
    // cells the arithmetic reads lie inside the patch; the clamp only keeps
    // every read inside the record
    const int di = min(max(i - i0, 0), w - 1), dj = min(max(j - j0, 0), w - 1);
    return __ldg(p + (int64_t)(dj * w + di) * stride);
  }
};

// subpixel_gauss3 (src/correlators.jl:499-520) with FP64 logarithms.
// (i, j) 0-based; returns 1-based refined (row, col).
// One axis: (ln Im - ln Ip) / (2 (ln Im - 2 ln I0 + ln Ip)), formed as
// ln(Im/Ip) / (2 ln(Im Ip / I0^2)) with the ratios in FP64 (exact products
// of floats, one rounding each): two logarithms instead of three.
__device__ __forceinline__ double gauss3_axis(float Im, float I0, float Ip) {
  if (!(Im > 0.f && I0 > 0.f && Ip > 0.f)) return 0.0;
  const double m = (double)Im, z = (double)I0, p = (double)Ip;
  const double den = log((m * p) / (z * z));
  return den != 0.0 ? log(m / p) / (2.0 * den) : 0.0;
}

template <class Acc> __device__ __forceinline__ void gauss3_fp64(const Acc& R, int nr, int nc, int i, int j, float* out) {
  double di = 0.0, dj = 0.0;
  const float I0 = R(i, j);
  if (i > 0 && i < nr - 1) di = gauss3_axis(R(i - 1, j), I0, R(i + 1, j));
  if (j > 0 && j < nc - 1) dj = gauss3_axis(R(i, j - 1), I0, R(i, j + 1));
  out[0] = (float)((double)(i + 1) + di);
  out[1] = (float)((double)(j + 1) + dj);
}

// subpixel_gauss9 (src/correlators.jl:534-564) with FP64 logarithms.
template <class Acc> __device__ __forceinline__ void gauss9_fp64(const Acc& R, int nr, int nc, int pr, int pc, float* out) {
  if (!(pr > 0 && pr < nr - 1 && pc > 0 && pc < nc - 1)) return gauss3_fp64(R, nr, nc, pr, pc, out);
  double sL = 0, sxL = 0, syL = 0, sxxL = 0, syyL = 0, sxyL = 0;
  for (int dj = -1; dj <= 1; ++dj)
    for (int di = -1; di <= 1; ++di) {
      float val = R(pr + di, pc + dj);
      if (!(val > 0.f)) return gauss3_fp64(R, nr, nc, pr, pc, out);
      double L = log((double)val);
      sL += L;
      sxL += dj * L;
      syL += di * L;
      sxxL += (dj * dj) * L;
      syyL += (di * di) * L;
      sxyL += (di * dj) * L;
    }
  double a1 = sxL / 6, a2 = syL / 6, a3 = sxxL / 2 - sL / 3, a4 = sxyL / 4, a5 = syyL / 2 - sL / 3;
  double D = 4 * a3 * a5 - a4 * a4;
  if (!(a3 < 0 && D > 0)) return gauss3_fp64(R, nr, nc, pr, pc, out);
  double dx = (a4 * a2 - 2 * a5 * a1) / D;
  double dy = (a4 * a1 - 2 * a3 * a2) / D;
  if (!(fabs(dx) <= 1 && fabs(dy) <= 1)) return gauss3_fp64(R, nr, nc, pr, pc, out);
  out[0] = (float)((double)(pr + 1) + dy);
  out[1] = (float)((double)(pc + 1) + dx);
}

// calculate_correlation_moment (src/quality.jl:49-74, neighbourhood 3):
// (c - pc)^2 in float like the Float32 reference, sums in FP64.
template <class Acc> __device__ __forceinline__ float moment_fp64(const Acc& R, int nr, int nc, float pr, float pc) {
  if (!(isfinite(pr) && isfinite(pc))) return __int_as_float(0x7fc00000);
  int r0 = (int)rintf(pr), c0 = (int)rintf(pc);  // 1-based, ties to even
  int rlo = max(1, r0 - 1), rhi = min(nr, r0 + 1), clo = max(1, c0 - 1), chi = min(nc, c0 + 1);
  if (rlo > rhi || clo > chi) return __int_as_float(0x7fc00000);
  // the 3 x 3 neighbourhood unrolled, clipped cells skipped: the loads issue
  // together and the sums keep the column-major order
  double sumC = 0, sdx = 0, sdy = 0;
#pragma unroll
  for (int dc = -1; dc <= 1; ++dc)
#pragma unroll
    for (int dr = -1; dr <= 1; ++dr) {
      const int c = c0 + dc, r = r0 + dr;
      if (c < clo || c > chi || r < rlo || r > rhi) continue;
      double w = fmax((double)R(r - 1, c - 1), 0.0);
      float dx = __fsub_rn((float)c, pc), dy = __fsub_rn((float)r, pr);
      sumC += w;
      sdx += (double)__fmul_rn(dx, dx) * w;
      sdy += (double)__fmul_rn(dy, dy) * w;
    }
  if (sumC < 1e-9) return __int_as_float(0x7fc00000);
  return (float)sqrt((sdx + sdy) / sumC);
}

struct PeakOut {
  float* du;
  float* dv;
  float* ratio;
  float* moment;
  float* alt_u;
  float* alt_v;
  int32_t nalt;
  int64_t G;
  float* packed;
  int32_t* locs;
};

// Peak record of one window (regional maxima), written by the correlation
// kernel in place of its epilogue and read by peak_epilogue_kernel: word w
// of job j at rec[w * njobs + j]. Words: 0 the number of peaks found (-1:
// window skipped), 1..K their values, then (row, col) per peak, then the
// 5 x 5 plane patch around the primary and a 3 x 3 patch around each
// alternative (column-major, cells outside the plane 0). A regional maximum
// is >= its neighbours, so its gauss3 offsets stay within 1/2 px and its
// gauss9 offsets within 1 px; the fits and the 3 x 3 moment around the
// refined primary therefore read only cells inside these patches.
__host__ __device__ constexpr int rec_words(int K) { return 17 + 12 * K; }
__device__ __forceinline__ int rec_patch(int K, int m) { return m == 0 ? 1 + 3 * K : 1 + 3 * K + 25 + 9 * (m - 1); }

// where the epilogue reads peak m's neighbourhood: the plane itself ...
struct PlaneSrc {
  const float* R;
  int ld;
  __device__ __forceinline__ PlaneAcc at(int, int, int) const { return PlaneAcc{R, ld}; }
};
struct BoxSrc {
  BoxAcc acc;
  __device__ __forceinline__ BoxAcc at(int, int, int) const { return acc; }
};
// ... or the patches of a peak record
struct RecSrc {
  const float* rec;  // rec + job
  int64_t stride;
  int K;
  __device__ __forceinline__ RecAcc at(int m, int pr, int pc) const {
    const int h = m == 0 ? 2 : 1;
    return RecAcc{rec + (int64_t)rec_patch(K, m) * stride, stride, pr - h, pc - h, 2 * h + 1};
  }
};

// The per-window outputs from the peaks found (analyze_plane!'s tail,
// src/correlators.jl:459-468): the primary refined by the chosen subpixel
// method, displacement from the plane centre, peak ratio and moment; the
// alternatives 1..npeaks-1 refined by gauss3; 1-based peak locations. Of the K
// peaks only [m0, m1) are handled (vals and locs[2 m0 ..] are read).
template <class Src>
__device__ void peak_outputs(const Src& src, int nr, int nc, int K, int npeaks, int subpixel, int nfound,
                             const float* vals, const int* locs, int64_t grid_id, int64_t job, const PeakOut& o,
                             int m0, int m1) {
  int found = 0;
  if (nfound > 0) {
    found = 1;
    while (found < nfound && vals[found] > 0.f) ++found;
  }
  const float NaN = __int_as_float(0x7fc00000);
  const int cr = nr / 2 + 1, cc = nc / 2 + 1;
  const int mmax = found < npeaks ? found : npeaks;  // peaks 1..mmax carry results
  float* pk = o.packed ? o.packed + job * (int64_t)(5 + 2 * (K - 1)) : nullptr;
  for (int m = m0; m < m1; ++m) {
    float ref[2] = {NaN, NaN};
    if (m < found && (m == 0 || m < mmax)) {
      const int pr = locs[2 * m], pc = locs[2 * m + 1];
      const auto R = src.at(m, pr, pc);
      if (m == 0 && subpixel == 1) gauss9_fp64(R, nr, nc, pr, pc, ref);
      else if (m == 0 && subpixel == 3) {
        ref[0] = (float)(pr + 1);
        ref[1] = (float)(pc + 1);
      } else gauss3_fp64(R, nr, nc, pr, pc, ref);
    }
    const float d_col = ref[1] - (float)cc, d_row = ref[0] - (float)cr;
    if (m == 0) {
      float ratio = NaN, mom = NaN;
      if (found > 0) {
        const float v1 = vals[0];
        ratio = found >= 2 ? v1 / vals[1] : (v1 > 0.f ? INFINITY : NaN);
        mom = moment_fp64(src.at(0, locs[0], locs[1]), nr, nc, ref[0], ref[1]);
      }
      if (grid_id >= 0 && o.du) {
        o.du[grid_id] = d_col;
        o.dv[grid_id] = d_row;
        o.ratio[grid_id] = ratio;
        o.moment[grid_id] = mom;
      }
      if (pk) {
        pk[0] = d_col;
        pk[1] = d_row;
        pk[2] = ratio;
        pk[3] = mom;
        pk[4] = (float)found;
      }
    } else {
      // alternative peak m (0-based): result only while m < min(found, npeaks)
      const bool has = m < mmax;
      const float au = has ? d_col : NaN, av = has ? d_row : NaN;
      if (grid_id >= 0 && o.alt_u && m - 1 < o.nalt) {
        o.alt_u[grid_id + (int64_t)(m - 1) * o.G] = au;
        o.alt_v[grid_id + (int64_t)(m - 1) * o.G] = av;
      }
      if (pk) {
        pk[5 + (m - 1)] = au;
        pk[5 + (K - 1) + (m - 1)] = av;
      }
    }
    if (o.locs) {
      int32_t* lc = o.locs + job * (int64_t)(2 * K);
      lc[2 * m] = m < found ? locs[2 * m] + 1 : 0;
      lc[2 * m + 1] = m < found ? locs[2 * m + 1] + 1 : 0;
    }
  }
}

// Peak analysis of one plane by a group of threads (tid in [0, gsize)).
// Every thread of the group must call this (uniform K and finder), because
// the merge synchronises the group.
// Only the box rows [rlo, rhi] x columns [clo, chi] can hold positive
// values (outside it the overlap gain is zero, so R is exactly 0 there); the
// scans cover it, plus the last pixel, the only place outside where a zero
// can be a regional maximum (every other pixel has a later neighbour >= 0).
// A thread's share of the box scan, fixed for a launch (the box and the
// group size do not change), so the integer divisions are done once:
// column strips of rps rows, S strips per column; this thread's first
// strip is column c, rows [r0, r1).
struct ScanPlan {
  int rlo, rhi, clo, chi;
  int bw, S, rps;
  int c, r0, r1;
};
__device__ __forceinline__ ScanPlan scan_plan(int gtid, int gsize, int rlo, int rhi, int clo, int chi) {
  ScanPlan sp;
  sp.rlo = rlo;
  sp.rhi = rhi;
  sp.clo = clo;
  sp.chi = chi;
  sp.bw = chi - clo + 1;
  sp.S = gsize / sp.bw > 0 ? gsize / sp.bw : 1;  // row segments per column
  sp.rps = (rhi - rlo + 1 + sp.S - 1) / sp.S;
  sp.c = clo + gtid % sp.bw;
  sp.r0 = rlo + (gtid / sp.bw) * sp.rps;
  sp.r1 = min(rhi + 1, sp.r0 + sp.rps);
  return sp;
}

// One column strip of the regional-maximum scan (src/localmax.jl:3-19): the
// 3x3 neighbourhood rolls down the strip in registers, rows r - 1 (t) and r
// (m) of the left, centre and right columns (3 loads per pixel). Earlier
// neighbours in column-major order (the left column and the pixel above)
// must not exceed the value, later ones (the right column and the pixel
// below) must stay below it; fmaxf drops NaN neighbours, which never block
// in the reference either.
template <bool BOXED> struct StripScan {
  const float* Cl;
  const float* Cc;
  const float* Cr;
  bool hl, hr;
  int c, r1;
  float lt, ct, rt, lm, cm, rm;
  // clo, chi, rlo: the box (BOXED: its outside is zero and not stored)
  static __device__ __forceinline__ float none() { return BOXED ? 0.f : __int_as_float(0x7fc00000); }
  __device__ __forceinline__ void init(const float* R, int ldr, int nc, int c_, int r0, int r1_, int clo, int chi,
                                       int rlo) {
    const float NaNf = none();
    c = c_;
    r1 = r1_;
    hl = c > (BOXED ? clo : 0);
    hr = c < (BOXED ? chi : nc - 1);
    Cc = R + c * ldr;
    Cl = hl ? Cc - ldr : Cc;
    Cr = hr ? Cc + ldr : Cc;
    lt = ct = rt = NaNf;
    if (r0 > (BOXED ? rlo : 0)) {
      lt = hl ? Cl[r0 - 1] : NaNf;
      ct = Cc[r0 - 1];
      rt = hr ? Cr[r0 - 1] : NaNf;
    }
    lm = hl ? Cl[r0] : NaNf;
    cm = Cc[r0];
    rm = hr ? Cr[r0] : NaNf;
  }
  // rows rb0 + 1 .. rb0 + SU of the three columns (NaN past the plane)
  // (past row rend: the box's or the plane's end)
  template <int SU> __device__ __forceinline__ void load(int rb0, int rend, float* l, float* m, float* r) const {
    const float NaNf = none();
#pragma unroll
    for (int u = 0; u < SU; ++u) {
      const int rr = rb0 + 1 + u;
      const bool ok = rr < rend;
      l[u] = ok && hl ? Cl[rr] : NaNf;
      m[u] = ok ? Cc[rr] : NaNf;
      r[u] = ok && hr ? Cr[rr] : NaNf;
    }
  }
  // tests row r (the centre value cm) and rolls down one row. A full list
  // rejects a key equal to its K-th: the strips of a thread reach the list in
  // index order, so a later index cannot win the tie.
  template <class TK>
  __device__ __forceinline__ void step(int r, float lb, float cb, float rbv, int nr, TK& tk, int K) {
    const float v = cm;
    if (r < r1 && !isnan(v)) {
      const uint32_t h = fkey(v);
      if (h > tk.thr) {
        const float e = fmaxf(fmaxf(lt, lm), fmaxf(lb, ct));
        const float l = fmaxf(fmaxf(rt, rm), fmaxf(rbv, cb));
        if (!(e > v) && !(l >= v)) tk.insert(h, ~(uint32_t)(r + c * nr), K);
      }
    }
    lt = lm;
    ct = cm;
    rt = rm;
    lm = lb;
    cm = cb;
    rm = rbv;
  }
};

// The regional maxima of an N x N plane of values >= 0 from its row maxima,
// for the fused kernels, whose last inverse pass holds whole rows (or N1
// columns of one) in registers: rmax[r] is the largest value of row r (as
// its bits, 0 for a row without one). A row maximum above those of both
// neighbouring rows belongs to a regional maximum (the last of its equals in
// the row), so the K-th largest of these is a lower bound of the K-th peak,
// and only pixels at or above it need the neighbour test. Few rows hold such
// pixels (the flanks of the strongest peaks: 5-8 of 31 at 32 points): they
// are read a row at a time, the pixels found are listed, and the lanes then
// test one each. With fewer than K such rows the bound is 0 and every pixel
// of the box is tested. A NaN neither blocks a neighbour nor is a peak, as
// in is_local_max; -0 does not occur. The lanes of a warp (or its half) take
// the rows lo + lane + j LANES; with several warps per plane each forms the
// bound by itself and reads every nwarps-th of the rows. list: room for
// 2 LANES entries per warp.
template <int N, int LANES, class TK>
__device__ __forceinline__ void scan_rows(TK& tk, const float* R, int ldr, int K, int lo, int hi, const uint32_t* rmax,
                                          uint16_t* list, int gtid, int nwarps) {
  constexpr int J = (N + LANES - 1) / LANES;
  const int lane = gtid & (LANES - 1), gwarp = gtid / LANES;
  const unsigned gm = grp_mask(LANES);
  const int sh = LANES < 32 ? (threadIdx.x & 31) & ~(LANES - 1) : 0;  // the group's first lane
  constexpr unsigned ALL = LANES < 32 ? (1u << (LANES & 31)) - 1u : 0xffffffffu;
  uint32_t M[J], cand[J];
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int r = lo + lane + j * LANES;
    M[j] = cand[j] = 0u;
    if (r <= hi) {
      M[j] = rmax[r];
      // rows outside the box are zero; a row outside the plane counts as one
      const uint32_t up = r > lo ? rmax[r - 1] : 0u, dn = r < hi ? rmax[r + 1] : 0u;
      cand[j] = M[j] > up && M[j] > dn ? M[j] : 0u;
    }
  }
  uint32_t thr = 0u;
  for (int k = 0; k < K; ++k) {  // equal candidates count once: the bound only gets lower
    uint32_t h = 0u;
#pragma unroll
    for (int j = 0; j < J; ++j) h = max(h, cand[j]);
    thr = __reduce_max_sync(gm, h);
    if (thr == 0u) break;
#pragma unroll
    for (int j = 0; j < J; ++j) cand[j] = cand[j] == thr ? 0u : cand[j];
  }
  // pixel e = r + c N of the list: a peak unless a neighbour blocks it
  // (neighbours outside the plane never do: NaN compares false)
  auto test = [&](int e) {
    const int r = e % N, c = e / N;
    const float* p = R + c * ldr + r;
    const float x = __int_as_float(0x7fc00000), v = *p;
    const bool hu = r > 0, hd = r < N - 1, hl = c > 0, hr = c < N - 1;
    const float ul = hu && hl ? p[-ldr - 1] : x, l = hl ? p[-ldr] : x, dl = hd && hl ? p[-ldr + 1] : x;
    const float u = hu ? p[-1] : x, d = hd ? p[1] : x;
    const float ur = hu && hr ? p[ldr - 1] : x, rt = hr ? p[ldr] : x, dr = hd && hr ? p[ldr + 1] : x;
    const float b = fmaxf(fmaxf(ul, l), fmaxf(dl, u)), t = fmaxf(fmaxf(ur, rt), fmaxf(dr, d));
    if (!isnan(v) && !(b > v) && !(t >= v)) tk.insert(fkey(v), ~(uint32_t)e, K);
  };
  list += gwarp * 2 * LANES;
  int cnt = 0, turn = 0;
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int base = lo + j * LANES;
    unsigned bits = (__ballot_sync(gm, base + lane <= hi && M[j] >= thr) >> sh) & ALL;
    while (bits) {
      const int r = base + __ffs(bits) - 1;
      bits &= bits - 1;
      if (nwarps > 1 && (turn++ % nwarps) != gwarp) continue;
      uint32_t v[J];
#pragma unroll
      for (int i = 0; i < J; ++i) {
        const int c = lo + lane + i * LANES;
        v[i] = c <= hi ? __float_as_uint(R[c * ldr + r]) : 0u;
      }
#pragma unroll
      for (int i = 0; i < J; ++i) {
        const int c = lo + lane + i * LANES;
        const bool in = c <= hi && v[i] >= thr;
        const unsigned b = (__ballot_sync(gm, in) >> sh) & ALL;
        if (in) list[cnt + __popc(b & ((1u << lane) - 1u))] = (uint16_t)(r + c * N);
        cnt += __popc(b);
        if (cnt >= LANES) {  // a full round of tests; the rest moves down
          __syncwarp(gm);
          test(list[lane]);
          const uint16_t q = list[LANES + lane];
          __syncwarp(gm);
          list[lane] = q;
          __syncwarp(gm);  // past the entries left, the next rows write these words again, by other lanes
          cnt -= LANES;
        }
      }
    }
  }
  __syncwarp(gm);
  if (lane < cnt) test(list[lane]);
}

// FN > 0: an FN x FN plane of a fused kernel with its row maxima (scan_rows);
// FN = 0: any plane, by column strips. BOXED: the plane is zero, and not
// stored, outside the box [rlo, rhi] x [clo, chi], which leaves at least the
// plane's last row and column out.
template <int KC, int FN, bool BOXED>
__device__ __forceinline__ void analyze_body(const float* R, int nr, int nc, int ldr, int K, int npeaks, int finder,
                                             int subpixel, int gtid, int gsize, uint32_t* red, bool active,
                                             float* s_vals, int* s_locs, int64_t grid_id, int64_t job,
                                             const PeakOut* o, bool poison, int bar, const ScanPlan sp,
                                             float* rec, int64_t rec_stride, const uint32_t* rmax = nullptr,
                                             uint16_t* list = nullptr) {
  const int rlo = sp.rlo, rhi = sp.rhi, clo = sp.clo, chi = sp.chi;
  // a poisoned plane (non-finite window data: the reference's plane is all
  // NaN there) yields no peak, so every output is NaN
  const bool scan = active && !poison;
  const int gwarp = gtid >> 5, nwarps = gsize >> 5;
  const int P = nr * nc;
  const BoxAcc box{R, ldr, rlo, rhi, clo, chi};
  auto at = [&](int i, int j) { return BOXED ? box(i, j) : R[j * ldr + i]; };
  int nfound = 0;
  if (finder == 0) {
    // regional maxima (src/localmax.jl:3-19): each thread walks column strips
    // of the box top to bottom (StripScan), keeping its K best in registers
    TopK<KC> tk;
    tk.init();
    if constexpr (FN > 0) {
      if (scan) scan_rows<FN, 32>(tk, R, ldr, K, rlo, rhi, rmax, list, gtid, nwarps);
    } else if (scan) {
      const int bw = sp.bw, S = sp.S, rps = sp.rps, ns = bw * S;
      // blocks of SU rows: the next SU rows of the three columns are loaded
      // together, so the loads of a block overlap instead of each row
      // waiting on its own
      constexpr int SU = 2;
      // strip `strip` of the box; an empty strip inside the box when it has
      // no rows (its addresses stay valid)
      auto strip_at = [&](int strip, int& c, int& r0, int& r1) {
        c = sp.c;
        r0 = sp.r0;
        r1 = sp.r1;
        if (strip != gtid) {  // a further strip: only when the box is wider than the group
          c = clo + strip % bw;
          r0 = rlo + (strip / bw) * rps;
          r1 = min(rhi + 1, r0 + rps);
        }
        if (strip >= ns || r0 >= r1) {
          c = clo;
          r0 = r1 = rlo;
        }
      };
      for (int strip = gtid; strip < ns; strip += gsize) {
        int c, r0, r1;
        strip_at(strip, c, r0, r1);
        if (r0 >= r1) continue;
        StripScan<BOXED> A;
        A.init(R, ldr, nc, c, r0, r1, clo, chi, rlo);
        for (int rb0 = r0; rb0 < r1; rb0 += SU) {
          float lb[SU], cb[SU], rbv[SU];  // rows rb0 + 1 .. rb0 + SU
          A.template load<SU>(rb0, BOXED ? rhi + 1 : nr, lb, cb, rbv);
#pragma unroll
          for (int u = 0; u < SU; ++u) A.step(rb0 + u, lb[u], cb[u], rbv[u], nr, tk, K);
        }
      }
    }
    if (scan && gtid == 0 && (rhi < nr - 1 || chi < nc - 1)) {  // the last pixel, outside the box
      const int r = nr - 1, c = nc - 1;
      if (BOXED) {  // a zero; its neighbours are zeros too but for a box that reaches the diagonal one
        if (!(at(r - 1, c - 1) > 0.f)) tk.insert(fkey(0.f), ~(uint32_t)(r + c * nr), K);
      } else if (is_local_max(R, nr, nc, ldr, r, c, R[c * ldr + r]))
        tk.insert(fkey(R[c * ldr + r]), ~(uint32_t)(r + c * nr), K);
    }
    // Merge: each warp takes its K best from its threads' lists by shuffle
    // rounds (lane m keeps the m-th); with several warps the warps' lists
    // meet in `red` behind one barrier and the first warp takes the group's
    // K best from them the same way.
    const int lane = gtid & 31;
    uint32_t mh = 0u, ml = 0u;
    int nw = warp_topk(tk, K, lane, mh, ml, grp_mask(gsize));
    if (nwarps > 1) {
      if (lane < K) {
        red[2 * (gwarp * K + lane)] = mh;
        red[2 * (gwarp * K + lane) + 1] = ml;
      }
      grp_sync(bar, gsize);
      if (gwarp == 0) {
        TopK<KC> tg;
        tg.init();
        for (int e = lane; e < nwarps * K; e += 32) {
          const uint32_t h = red[2 * e], l = red[2 * e + 1];
          if (h != 0u) tg.insert(h, l, K);
        }
        nw = warp_topk(tg, K, lane, mh, ml, 0xffffffffu);
      }
    }
    if (gwarp == 0) {
      nfound = nw;
      if (lane < nw) {
        const int lin = (int)(~ml);
        s_vals[lane] = at(lin % nr, lin / nr);
        s_locs[2 * lane] = lin % nr;
        s_locs[2 * lane + 1] = lin / nr;
      }
    }
  } else {
    // exclusion finder (src/correlators.jl:390-421): K scans, box +-2
    bool done = false;
    for (int round = 0; round < K; ++round) {  // every round runs: group_argmax synchronises the group
      // the box first; when its best is not positive the maximum can lie
      // outside it (a zero earlier in column-major order), so rescan all
      uint32_t whi = 0u, wlo = 0u;
      for (int pass = 0; pass < 2; ++pass) {
        const int bw = chi - clo + 1, bht = rhi - rlo + 1;
        const int n = pass == 0 ? bw * bht : P;
        uint32_t bh = 0u, bl = 0u;
        if (scan && !done) {
          for (int t = gtid; t < n; t += gsize) {
            const int r = pass == 0 ? rlo + t % bht : t % nr, c = pass == 0 ? clo + t / bht : t / nr;
            bool ex = false;
            for (int q = 0; q < nfound; ++q)
              if (abs(r - s_locs[2 * q]) <= 2 && abs(c - s_locs[2 * q + 1]) <= 2) { ex = true; break; }
            if (ex) continue;
            const float v = at(r, c);
            if (!(v > -INFINITY)) continue;  // NaN and -Inf never beat the initial -Inf
            const uint32_t h = fkey(v), l = ~(uint32_t)(r + c * nr);
            if (h > bh || (h == bh && l > bl)) { bh = h; bl = l; }
          }
        }
        group_argmax(bh, bl, red, gwarp, gsize, whi, wlo, bar);
        if (whi > fkey(0.f) || (rlo == 0 && clo == 0 && rhi == nr - 1 && chi == nc - 1)) break;  // positive, or the box is the plane
      }
      if (!done && whi != 0u) {
        const int lin = (int)(~wlo);
        const float best = at(lin % nr, lin / nr);
        if (nfound > 0 && !(best > 0.f)) {
          done = true;  // secondary peaks must be positive
        } else {
          if (gtid == 0) {
            s_vals[nfound] = best;
            s_locs[2 * nfound] = lin % nr;
            s_locs[2 * nfound + 1] = lin / nr;
          }
          ++nfound;
        }
      } else {
        done = true;
      }
      grp_sync(bar, gsize);  // s_locs visible to the next round's exclusion test
    }
  }
  // Epilogue on the group's first warp, after the last merge step wrote
  // s_vals / s_locs: with a record buffer (regional maxima) the lanes of the
  // peaks store the peak record and peak_epilogue_kernel forms the outputs;
  // otherwise lane 0 forms them here.
  if (gtid >= 32 || !active) return;
  __syncwarp(grp_mask(gsize));
  if (rec && finder == 0) {
    // the record's words spread over the lanes (a few each), so its shared
    // loads and global stores overlap instead of one lane walking the patches
    const int lanes = gsize < 32 ? gsize : 32, base0 = 1 + 3 * K, nw = rec_words(K);
    for (int wd = gtid; wd < nw; wd += lanes) {
      float val = 0.f;
      if (wd == 0) {
        val = __int_as_float(nfound);
      } else if (wd <= K) {
        val = wd - 1 < nfound ? s_vals[wd - 1] : 0.f;
      } else if (wd < base0) {
        const int m = (wd - 1 - K) >> 1;
        val = m < nfound ? __int_as_float(s_locs[wd - 1 - K]) : 0.f;
      } else {
        const int e = wd - base0;  // primary: 25 cells; alternative m: 9 cells
        const int m = e < 25 ? 0 : 1 + (e - 25) / 9, cell = e < 25 ? e : (e - 25) % 9;
        const int h = m == 0 ? 2 : 1, w = 2 * h + 1;
        if (m < nfound) {
          const int i = s_locs[2 * m] + cell % w - h, j = s_locs[2 * m + 1] + cell / w - h;
          val = (i >= 0 && i < nr && j >= 0 && j < nc) ? at(i, j) : 0.f;
        }
      }
      rec[(int64_t)wd * rec_stride + job] = val;
    }
    return;
  }
  if (gtid == 0) {
    if constexpr (BOXED)
      peak_outputs(BoxSrc{{R, ldr, rlo, rhi, clo, chi}}, nr, nc, K, npeaks, subpixel, nfound, s_vals, s_locs, grid_id, job, *o, 0, K);
    else
      peak_outputs(PlaneSrc{R, ldr}, nr, nc, K, npeaks, subpixel, nfound, s_vals, s_locs, grid_id, job, *o, 0, K);
  }
}

// The analysis as a call: small planes keep it out of line (the kernel's
// transform stages then keep their registers); large planes inline it.
template <int FN = 0, bool BOXED = false>
__device__ __noinline__ void analyze_group(const float* R, int nr, int nc, int ldr, int K, int npeaks, int finder,
                                           int subpixel, int gtid, int gsize, uint32_t* red, bool active,
                                           float* s_vals, int* s_locs, int64_t grid_id, int64_t job,
                                           const PeakOut* o, bool poison, int bar, const ScanPlan sp,
                                           float* rec, int64_t rec_stride, const uint32_t* rmax = nullptr,
                                           uint16_t* list = nullptr) {
  if (K <= 4)
    analyze_body<4, FN, BOXED>(R, nr, nc, ldr, K, npeaks, finder, subpixel, gtid, gsize, red, active, s_vals, s_locs,
                               grid_id, job, o, poison, bar, sp, rec, rec_stride, rmax, list);
  else
    analyze_body<KMAX, FN, BOXED>(R, nr, nc, ldr, K, npeaks, finder, subpixel, gtid, gsize, red, active, s_vals, s_locs,
                                  grid_id, job, o, poison, bar, sp, rec, rec_stride, rmax, list);
}

// S(k) = conj(FA(k)) FB(k) of the packed transform Z = F(a + i b), from
// X = Z(k) and Zm = Z(-k): FA = (X + conj(Zm))/2, FB = (X - conj(Zm))/(2i)
// (spectrum!, src/correlators.jl:266-279); the phase method divides by
// |S| + eps(Float32) and applies the spectral filter weight wk.
__device__ __forceinline__ float2 cross_spectrum(float2 X, float2 Zm, int method, float wk) {
  const float2 s = cadd2(X, Zm), d = csub2(X, Zm);
  const float Ar = 0.5f * s.x, Ai = 0.5f * d.y;
  const float Br = 0.5f * s.y, Bi = -0.5f * d.x;
  float2 S = cmul(make_float2(Ar, -Ai), make_float2(Br, Bi));
  if (method == 1) {
    const float den = hypotf(S.x, S.y) + 1.1920929e-7f;
    S = make_float2((wk * S.x) / den, (wk * S.y) / den);
  }
  return S;
}

}  // namespace hh
