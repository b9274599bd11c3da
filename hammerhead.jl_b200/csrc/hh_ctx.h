// Library context and host-side helpers shared by the C-ABI translation units
// (hh_api.cu: single-pair schedule and hooks; hh_batch.cu: batched schedule).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <sstream>
#include <string>
#include <tuple>
#include <vector>

#include "hammerhead_b200.h"
#include "hh_internal.h"

using hh::CorrArgs;

namespace hhd {

inline thread_local std::string g_err;  // context-free failures

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

struct TableKey {
  int wr, wc, sr, sc, apod, method, padded;
  bool operator<(const TableKey& o) const {
    return std::tie(wr, wc, sr, sc, apod, method, padded) < std::tie(o.wr, o.wc, o.sr, o.sc, o.apod, o.method, o.padded);
  }
};
struct Tables {
  float* apod = nullptr;
  float* gain = nullptr;
  float* phasew = nullptr;
  // support of the gain, or the kept search lags, in fftshifted rows/columns (0, 0: whole plane)
  int box_lo = 0, box_hi = 0;
  // the same per axis for any plane shape (fftshifted rows rlo..rhi,
  // columns clo..chi; the whole plane when there is no gain or lag limit)
  int rlo = 0, rhi = -1, clo = 0, chi = -1;
};

}  // namespace hhd

struct hh_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 148;
  std::string err;
  std::map<std::string, hhd::DevBuf> bufs;
  std::map<hhd::TableKey, hhd::Tables> tables;
  std::map<int64_t, std::pair<float*, float*>> bs_factors;  // line length -> (cp, inv)
  float* pinned = nullptr;  // page-locked block (HH_PINNED_BYTES) for scalars and small results
  // staged pair for the hook-level entry points
  int64_t nr = 0, nc = 0;
  const float* curA = nullptr;
  const float* curB = nullptr;
  bool staged = false;
  const uint8_t* hook_mask = nullptr;  // image mask of the hook calls (hh_stage_mask), device
  // host-side allocation-failure injection (hh_debug_fail_alloc): the
  // allocation attempt that brings the count to zero fails with HH_ERR_OOM
  // as a failing cudaMalloc would; negative = off
  int64_t fail_alloc_after = -1;
  // timing of the last schedule
  std::vector<float> pass_ms;
  std::vector<int32_t> pass_sweeps;
  std::vector<cudaEvent_t> events;
  // kernel accounting (hh_set_profiling / hh_profile_read / hh_launch_count)
  bool prof = false;
  struct Pending {
    int cls;
    cudaEvent_t a, b;
    double flops, bytes;
    int64_t units, nk;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> evpool;
  hh_kernel_profile acc[HH_K_CLASSES] = {};
  int64_t launches = 0;
  // batched-schedule plans by batch shape (hh_batch.cu), most recent last
  std::vector<std::pair<std::string, void*>> bplans;
  void (*bplan_free)(void*) = nullptr;
  // cross-process reduction of the ensemble sums (hh_set_ensemble_reducer)
  hh_ensemble_reducer ens_reduce = nullptr;
  void* ens_reduce_user = nullptr;
  // correlation kernel CTA shape per (FFT size, data extent), from
  // hh_set_corr_variant / hh_autotune_correlation (absent: 0, the default)
  std::map<std::pair<int, int>, int> corr_var;
  // general-shape correlation: twiddle tables exp(-2 pi i t / n) by length
  std::map<int, float2*> gc_twiddles;
};

namespace hhd {

// Page-locked block of a context: a result of up to 40 k vectors comes back
// through it in one copy instead of one pageable copy per field (8-10 us each).
constexpr size_t HH_PINNED_BYTES = 1 << 20;

inline hh_status fail(hh_ctx* ctx, hh_status code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  else g_err = msg;
  return code;
}

#define HH_CK(call)                                                                                  \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess)                                                                           \
      return fail(ctx, e_ == cudaErrorMemoryAllocation ? HH_ERR_OOM : HH_ERR_CUDA,                   \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                               \
  } while (0)

#define HH_TRY(expr)                  \
  do {                                \
    hh_status s_ = (expr);            \
    if (s_ != HH_OK) return s_;       \
  } while (0)

inline std::string tup(const int32_t* t) {
  std::ostringstream o;
  o << "(" << t[0] << ", " << t[1] << ")";
  return o.str();
}
inline std::string num(double x) {
  std::ostringstream o;
  o << x;
  return o.str();
}

// cudaMalloc through the context, with the injected failure of
// hh_debug_fail_alloc (no device call is made for an injected failure).
inline cudaError_t ctx_malloc(hh_ctx* ctx, void** p, size_t bytes) {
  if (ctx && ctx->fail_alloc_after >= 0 && ctx->fail_alloc_after-- == 0) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMalloc(p, bytes);
}

// Device buffer by name, grown on demand (never shrunk): a steady state of
// equally sized calls allocates nothing.
template <class T> hh_status buf(hh_ctx* ctx, const char* name, size_t count, T** out) {
  DevBuf& b = ctx->bufs[name];
  const size_t need = std::max<size_t>(count, 1) * sizeof(T);
  if (b.bytes < need) {
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
    cudaError_t e = ctx_malloc(ctx, &b.p, need);
    if (e != cudaSuccess)
      return fail(ctx, HH_ERR_OOM, std::string("device allocation of ") + std::to_string(need) + " bytes for " + name +
                                       " failed: " + cudaGetErrorString(e));
    b.bytes = need;
  }
  *out = static_cast<T*>(b.p);
  return HH_OK;
}

// ---------------------------------------------------------------------------
// Host grid: pass_grid (src/pipeline.jl:529-555)
struct Grid {
  int ny = 0, nx = 0;
  hh::WinGrid win{};  // where its windows lie
  std::vector<float> x, y;
  std::vector<uint8_t> gmask;
  std::vector<int32_t> jobs;  // 0-based gi, gj, rs, cs
  bool any_mask = false;
  int64_t G() const { return (int64_t)ny * nx; }
};

// The grid without its mask and window list.
inline hh_status grid_axes(hh_ctx* ctx, int64_t nr, int64_t nc, const hh_pass_desc& p, Grid& g) {
  const int wr = p.window[0], wc = p.window[1], sr = p.search[0], sc = p.search[1];
  const int mr = (sr - wr) / 2, mc = (sc - wc) / 2;
  if (sr > nr || sc > nc)
    return fail(ctx, HH_ERR_ARG, "search area " + tup(p.search) + " exceeds image size (" + std::to_string(nr) + ", " +
                                     std::to_string(nc) + ")");
  g.win = hh::WinGrid{mr, wr - p.overlap[0], mc, wc - p.overlap[1]};
  g.ny = (int)((nr - wr - 2 * mr) / g.win.rstep + 1);
  g.nx = (int)((nc - wc - 2 * mc) / g.win.cstep + 1);
  g.x.resize(g.nx);
  g.y.resize(g.ny);
  for (int j = 0; j < g.nx; ++j) g.x[j] = (float)((double)(mc + 1 + (int64_t)j * g.win.cstep) + (wc - 1) / 2.0);
  for (int i = 0; i < g.ny; ++i) g.y[i] = (float)((double)(mr + 1 + (int64_t)i * g.win.rstep) + (wr - 1) / 2.0);
  g.any_mask = false;
  return HH_OK;
}

// The window list of the cells that gmask leaves.
inline void grid_jobs(Grid& g) {
  g.jobs.clear();
  g.jobs.reserve(4 * (size_t)g.G());
  for (int gj = 0; gj < g.nx; ++gj)
    for (int gi = 0; gi < g.ny; ++gi)
      if (!g.gmask[gi + (size_t)gj * g.ny]) {
        const int32_t q[4] = {gi, gj, g.win.r0 + gi * g.win.rstep, g.win.c0 + gj * g.win.cstep};
        g.jobs.insert(g.jobs.end(), q, q + 4);
      }
}

inline hh_status make_grid(hh_ctx* ctx, int64_t nr, int64_t nc, const hh_pass_desc& p, const uint8_t* mask, double thr,
                    Grid& g) {
  HH_TRY(grid_axes(ctx, nr, nc, p, g));
  const int wr = p.window[0], wc = p.window[1], sr = p.search[0], sc = p.search[1];
  const int mr = (sr - wr) / 2, mc = (sc - wc) / 2;
  g.gmask.assign((size_t)g.ny * g.nx, 0);
  if (mask) {
    for (int gj = 0; gj < g.nx; ++gj)
      for (int gi = 0; gi < g.ny; ++gi) {
        const int64_t rs = g.win.r0 + (int64_t)gi * g.win.rstep, cs = g.win.c0 + (int64_t)gj * g.win.cstep;
        int64_t cw = 0, csr = 0;
        for (int j = 0; j < wc; ++j)
          for (int i = 0; i < wr; ++i) cw += mask[(rs + i) + (cs + j) * nr] != 0;
        const int64_t srs = rs - mr, scs = cs - mc;
        for (int j = 0; j < sc; ++j)
          for (int i = 0; i < sr; ++i) csr += mask[(srs + i) + (scs + j) * nr] != 0;
        const double fw = (double)cw / (double)(wr * wc), fs = (double)csr / (double)(sr * sc);
        const uint8_t m = fw >= thr || fs >= thr;
        g.gmask[gi + (size_t)gj * g.ny] = m;
        g.any_mask |= m != 0;
      }
  }
  grid_jobs(g);
  return HH_OK;
}

inline int fft_size(const hh_pass_desc& p) { return p.padding ? 2 * p.search[0] : p.search[0]; }
inline int fft_rows(const hh_pass_desc& p) { return p.padding ? 2 * p.search[0] : p.search[0]; }
inline int fft_cols(const hh_pass_desc& p) { return p.padding ? 2 * p.search[1] : p.search[1]; }

// A fused shared-memory kernel exists for this pass (square window and
// search area of a specialised size); otherwise the general-shape kernel runs.
inline bool corr_special(const hh_pass_desc& p) {
  return p.window[0] == p.window[1] && p.search[0] == p.search[1] && hh::correlate_supported(fft_size(p), p.search[0]);
}

// The CTA shape chosen for a pass's correlation launches.
inline int32_t corr_variant(const hh_ctx* ctx, const hh_pass_desc& p) {
  auto it = ctx->corr_var.find({fft_size(p), (int)p.search[0]});
  return it == ctx->corr_var.end() ? 0 : it->second;
}

// apodization_window (src/correlators.jl:18-25), computed in double like
// Julia: centre (w + 1)/2 and sigma w/4 per axis, wr x wc column-major
inline void apod_table(int wr, int wc, int apod, std::vector<float>& out) {
  out.assign((size_t)wr * wc, 1.0f);
  if (apod == HH_APOD_NONE) return;
  const double cr = (wr + 1) / 2.0, cc = (wc + 1) / 2.0, sr = wr / 4.0, sc = wc / 4.0;
  for (int j = 1; j <= wc; ++j)
    for (int i = 1; i <= wr; ++i)
      out[(i - 1) + (size_t)(j - 1) * wr] =
          (float)std::exp(-((i - cr) * (i - cr) / (2 * sr * sr) + (j - cc) * (j - cc) / (2 * sc * sc)));
}

// overlap gain (src/correlators.jl:170-181): the weight of each lag is the
// autocorrelation of the apodization window (the reference forms it with an
// FFT in T); gain = wmax / w where w >= wmax / 2, else 0, in the fftshifted
// layout of the 2wr x 2wc plane. Square windows up to 64 px sum the float
// window's products directly in double; larger or rectangular windows use
// the separable form of the same window (the product of the row and column
// autocorrelations of the double-precision factors), the same quantity to
// within the float rounding of the window values.
inline void gain_table(int wr, int wc, int apod, const std::vector<float>& ap, std::vector<float>& out) {
  const int NR = 2 * wr, NC = 2 * wc;
  std::vector<float> wt((size_t)NR * NC, 0.f);
  if (wr == wc && wr <= 64) {
    const int W = wr, N = NR;
    for (int qs = 0; qs < N; ++qs)
      for (int ps = 0; ps < N; ++ps) {
        const int dp = ps - N / 2, dq = qs - N / 2;
        if (std::abs(dp) >= W || std::abs(dq) >= W) continue;
        double acc = 0;
        for (int q = std::max(0, -dq); q < std::min(W, W - dq); ++q)
          for (int p = std::max(0, -dp); p < std::min(W, W - dp); ++p)
            acc += (double)ap[p + (size_t)q * W] * (double)ap[(p + dp) + (size_t)(q + dq) * W];
        wt[ps + (size_t)qs * N] = (float)std::fabs(acc);
      }
  } else {
    auto axis = [apod](int w, std::vector<double>& ac) {
      std::vector<double> g(w, 1.0);
      if (apod == HH_APOD_GAUSS) {
        const double c = (w + 1) / 2.0, s = w / 4.0;
        for (int i = 1; i <= w; ++i) g[i - 1] = std::exp(-(i - c) * (i - c) / (2 * s * s));
      }
      ac.assign(2 * w, 0.0);  // lag d at index d + w
      for (int d = -(w - 1); d <= w - 1; ++d) {
        double a = 0;
        for (int i = std::max(0, -d); i < std::min(w, w - d); ++i) a += g[i] * g[i + d];
        ac[d + w] = a;
      }
    };
    std::vector<double> ar, acol;
    axis(wr, ar);
    axis(wc, acol);
    for (int qs = 0; qs < NC; ++qs)
      for (int ps = 0; ps < NR; ++ps) {
        const int dp = ps - NR / 2, dq = qs - NC / 2;
        if (std::abs(dp) >= wr || std::abs(dq) >= wc) continue;
        wt[ps + (size_t)qs * NR] = (float)std::fabs(ar[dp + wr] * acol[dq + wc]);
      }
  }
  float wmax = 0.f;
  for (float w : wt) wmax = std::max(wmax, w);
  out.resize(wt.size());
  for (size_t k = 0; k < wt.size(); ++k) out[k] = wt[k] >= wmax / 2 ? wmax / wt[k] : 0.f;
}

// PhaseCorrelator Gaussian spectral filter (src/correlators.jl:96-129):
// fftfreq bins of each axis, sigma = min(nr, nc) / 8, natural FFT order
inline void phase_table(int NR, int NC, std::vector<float>& out) {
  out.resize((size_t)NR * NC);
  const double fs = std::min(NR, NC) / 8.0;
  for (int j = 0; j < NC; ++j)
    for (int i = 0; i < NR; ++i) {
      const double fi = i < (NR + 1) / 2 ? i : i - NR, fj = j < (NC + 1) / 2 ? j : j - NC;
      out[i + (size_t)j * NR] = (float)std::exp(-(fi * fi + fj * fj) / (2 * fs * fs));
    }
}

inline hh_status get_tables(hh_ctx* ctx, const hh_pass_desc& p, Tables& t) {
  const int wr = p.window[0], wc = p.window[1], sr = p.search[0], sc = p.search[1];
  const int NR = fft_rows(p), NC = fft_cols(p);
  TableKey key{wr, wc, sr, sc, p.apodization, p.method, p.padding};
  auto it = ctx->tables.find(key);
  if (it != ctx->tables.end()) {
    t = it->second;
    return HH_OK;
  }
  std::vector<float> ap, gn, ph;
  apod_table(wr, wc, p.apodization, ap);
  Tables nt;
  nt.rhi = NR - 1;
  nt.chi = NC - 1;
  HH_CK(cudaMalloc(&nt.apod, ap.size() * sizeof(float)));
  HH_CK(cudaMemcpy(nt.apod, ap.data(), ap.size() * sizeof(float), cudaMemcpyHostToDevice));
  if (sr != wr || sc != wc) {
    // enlarged search area: no overlap gain (CrossCorrelator, src/correlators.jl:73);
    // only lags with |lag| <= (S - W) / 2 are kept (restrict_search_lags!, :347-355)
    nt.rlo = NR / 2 - (sr - wr) / 2;
    nt.rhi = NR / 2 + (sr - wr) / 2;
    nt.clo = NC / 2 - (sc - wc) / 2;
    nt.chi = NC / 2 + (sc - wc) / 2;
    if (NR == NC && sr == sc && wr == wc) {
      const int m = (sr - wr) / 2;
      nt.box_lo = NR / 2 - m;
      nt.box_hi = NR / 2 + m;
    }
  } else if (p.padding) {
    gain_table(wr, wc, p.apodization, ap, gn);
    {  // bounding rows and columns of the nonzero gain
      int rl = NR, rh = -1, cl = NC, ch = -1;
      for (int q = 0; q < NC; ++q)
        for (int r = 0; r < NR; ++r)
          if (gn[r + (size_t)q * NR] != 0.f) {
            rl = std::min(rl, r);
            rh = std::max(rh, r);
            cl = std::min(cl, q);
            ch = std::max(ch, q);
          }
      if (rh >= 0) {
        nt.rlo = rl;
        nt.rhi = rh;
        nt.clo = cl;
        nt.chi = ch;
      }
    }
    if (NR == NC) {
      // bounding box of the nonzero gain (square and centred, by symmetry)
      int lo = NR, hi = -1;
      for (int q = 0; q < NC; ++q)
        for (int r = 0; r < NR; ++r)
          if (gn[r + (size_t)q * NR] != 0.f) {
            lo = std::min(lo, std::min(r, q));
            hi = std::max(hi, std::max(r, q));
          }
      if (hi > 0) {
        nt.box_lo = lo;
        nt.box_hi = hi;
      }
    }
    HH_CK(cudaMalloc(&nt.gain, gn.size() * sizeof(float)));
    HH_CK(cudaMemcpy(nt.gain, gn.data(), gn.size() * sizeof(float), cudaMemcpyHostToDevice));
  }
  if (p.method == HH_PHASE) {
    phase_table(NR, NC, ph);
    HH_CK(cudaMalloc(&nt.phasew, ph.size() * sizeof(float)));
    HH_CK(cudaMemcpy(nt.phasew, ph.data(), ph.size() * sizeof(float), cudaMemcpyHostToDevice));
  }
  ctx->tables[key] = nt;
  t = nt;
  return HH_OK;
}

// Twiddle table exp(-2 pi i t / n), t = 0 .. n-1, of one FFT length, built
// once per context (double-precision angles, each entry rounded once).
inline hh_status gc_twiddles(hh_ctx* ctx, int n, const float2** out) {
  auto it = ctx->gc_twiddles.find(n);
  if (it == ctx->gc_twiddles.end()) {
    std::vector<float2> h(n);
    for (int t = 0; t < n; ++t) {
      // the angle in double (relative error ~1e-16, far below float rounding)
      const double a = -2.0 * M_PI * (double)t / (double)n;
      h[t] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    float2* d = nullptr;
    HH_CK(cudaMalloc(&d, (size_t)n * sizeof(float2)));
    HH_CK(cudaMemcpy(d, h.data(), (size_t)n * sizeof(float2), cudaMemcpyHostToDevice));
    it = ctx->gc_twiddles.emplace(n, d).first;
  }
  *out = it->second;
  return HH_OK;
}

// Shared memory of the general kernel's two line buffers (at most this much)
constexpr size_t GC_SMEM_LINES = 192 * 1024;
// planes the general kernel accepts (complex + real plane per CTA slice)
constexpr int64_t GC_MAX_POINTS = (int64_t)1 << 22;

// FFT lengths the general kernel transforms in registers (16 x B, two lines per warp)
inline bool gc_reg_length(int n) { return n == 32 || n == 64 || n == 128 || n == 256; }

// Is the pass's FFT shape one the general kernel can run?
inline bool gcorr_shape_ok(const hh_pass_desc& p) {
  int8_t rr[24];
  const int NR = fft_rows(p), NC = fft_cols(p);
  return NR >= 2 && NC >= 2 && (int64_t)NR * NC <= GC_MAX_POINTS && hh::gcorr_radix_plan(NR, rr) > 0 &&
         hh::gcorr_radix_plan(NC, rr) > 0 && 2 * (size_t)(NC + 16) * 2 * sizeof(float2) <= GC_SMEM_LINES &&
         2 * 2 * (size_t)(NR + 16) * sizeof(float2) <= GC_SMEM_LINES;
}

// Fill the general-shape fields of a correlation launch: shapes, radix
// plans, twiddles, chunking and the scratch slice geometry (one slice per
// CTA) for ca.njobs windows; gcorr_prepare also points it at the context's
// scratch buffer (grown on demand), a batched plan at its own.
inline hh_status gcorr_setup(hh_ctx* ctx, const hh_pass_desc& p, CorrArgs& ca) {
  ca.wr = p.window[0];
  ca.wc = p.window[1];
  ca.sr = p.search[0];
  ca.sc = p.search[1];
  ca.nfr = fft_rows(p);
  ca.nfc = fft_cols(p);
  ca.gc_nst_r = hh::gcorr_radix_plan(ca.nfr, ca.gc_radix_r);
  ca.gc_nst_c = hh::gcorr_radix_plan(ca.nfc, ca.gc_radix_c);
  if (ca.gc_nst_r < 0 || ca.gc_nst_c < 0 || !gcorr_shape_ok(p))
    return fail(ctx, HH_ERR_UNSUPPORTED,
                "backend :b200 has no correlation kernel for an FFT plane of " + std::to_string(ca.nfr) + " x " +
                    std::to_string(ca.nfc));
  HH_TRY(gc_twiddles(ctx, ca.nfr, &ca.twr));
  HH_TRY(gc_twiddles(ctx, ca.nfc, &ca.twc));
  Tables tb;
  HH_TRY(get_tables(ctx, p, tb));
  ca.gc_box[0] = tb.rlo;
  ca.gc_box[1] = tb.rhi;
  ca.gc_box[2] = tb.clo;
  ca.gc_box[3] = tb.chi;
  // columns passes: per warp one line (two, one per half-warp, for the
  // register-form lengths 32..256), two buffers per line, as many warps as
  // fit; rows pass: chunks of row pairs, two buffers each, at most two lines
  // per warp. Lines are staged with 16 elements of padding (the register
  // form's exchange). The complex plane holds the data columns, later the
  // box's, the real plane the box.
  const size_t ldr = (size_t)ca.nfr + 16, ldc = (size_t)ca.nfc + 16;
  const int lpw = gc_reg_length(ca.nfr) ? 2 : 1;
  const int64_t nboxc = tb.chi - tb.clo + 1, ldb = (tb.rhi - tb.rlo + 1) | 1;
  const int64_t zf = std::max<int64_t>(p.search[1], nboxc) * ca.nfr;  // float2
  const size_t planes = (size_t)zf * sizeof(float2) + (size_t)(nboxc * ldb) * sizeof(float);
  // An SM has 228 KB of shared memory, 1 KB of it taken per CTA, and registers
  // for 6, 2 or 1 CTAs of 128, 256 or 512 threads. The smallest CTA whose
  // planes leave room for 4, 2 or 1 of it: a window is then slower, but several
  // cover each other's barriers (6 CTAs of 128 threads against 4: 0.33 and
  // 0.35 ms for 8001 windows of 24 x 16, padded).
  constexpr size_t SM = 228 * 1024, CTA = 1024;
  int per_sm = 0;
  for (int t : {128, 256, 512}) {
    const size_t b = hh::gcorr_plane_smem(ca.nfr, ca.nfc, tb.rhi - tb.rlo + 1, nboxc, t);
    if (b > SM * t / 512 - CTA) continue;
    per_sm = t == 128 ? std::min<int>(hh::gcorr_plane_ctas, (int)(SM / (b + CTA))) : 512 / t;
    ca.gc_threads = t;
    ca.gc_in_smem = 1;
    ca.gc_smem_bytes = b;
    break;
  }
  if (!per_sm) {
    // Planes that fit no CTA's shared memory go to L2, one CTA of 512 threads
    // per SM. Two CTAs of 256 cover each other's waits where both lengths are
    // transformed in registers, the line buffers fit twice and the slices
    // together stay within L2: with 4000 windows of 256 x 256 points 4.28
    // against 4.64 ms, of 128 x 256 2.39 and 2.69; other lengths gain nothing
    // (280 x 216, 880 windows: 4.24 and 4.28 ms; 122 x 122: 60.5 and 58.4). But
    // a window takes 1.3 times as long on 256 threads even where it has the SM
    // for itself, so a round of one window per SM is left to 512: at 256 x 256
    // 148 windows 226 us on 256 threads and 176 on 512, 290: 324 and 342, 440:
    // 627 and 508, 740: 932 and 842, 961: 1108 and 1171, 1036: 1237 and 1175.
    auto shape = [&](int threads) {
      const int warps = threads / 32;
      ca.gc_threads = threads;
      ca.gc_in_smem = 0;
      ca.gc_col_warps = std::max(1, std::min(warps, (int)(GC_SMEM_LINES / (2 * lpw * ldr * sizeof(float2)))));
      ca.gc_chunk_c = std::max(2, std::min(2 * warps, (int)(GC_SMEM_LINES / (2 * ldc * sizeof(float2)))) & ~1);
      const size_t lines = std::max((size_t)ca.gc_col_warps * lpw * ldr, (size_t)ca.gc_chunk_c * ldc);
      ca.gc_smem_lines = (int64_t)(2 * lines * sizeof(float2));
      ca.gc_smem_bytes = ca.gc_smem_lines + hh::gcorr_smem_extra(warps);
      return (size_t)ca.gc_smem_bytes;
    };
    const int64_t sms = ctx->num_sms, last = ca.njobs % (2 * sms);  // windows of the last round of two per SM
    const bool single = ca.njobs <= sms || (ca.njobs <= 7 * sms && last > sms / 2 && last <= sms);
    per_sm = 2;
    if (single || lpw == 1 || !gc_reg_length(ca.nfc) || shape(256) > SM / 2 - CTA || 2 * sms * planes > (size_t)110 << 20) {
      per_sm = 1;
      shape(512);
    }
  }
  ca.gscr_slices = per_sm * ctx->num_sms;
  ca.gscr_stride = ca.gc_in_smem ? 0 : (zf + (nboxc * ldb + 1) / 2 + 31) & ~(int64_t)31;  // 256-byte aligned slices
  return HH_OK;
}
inline hh_status gcorr_prepare(hh_ctx* ctx, const hh_pass_desc& p, CorrArgs& ca) {
  HH_TRY(gcorr_setup(ctx, p, ca));
  if (ca.gc_in_smem) return HH_OK;
  return buf(ctx, "gcorr_scratch", (size_t)ca.gscr_slices * ca.gscr_stride, &ca.gscr);
}

// The window shape of an uncertainty launch (rows W, columns Wc), and for
// rectangular or large windows the general form's scratch slices (one per
// CTA; the buffer is the context's and grows on demand).
inline void uq_setup(hh_ctx* ctx, int wr, int wc, hh::UQArgs& ua) {
  ua.W = wr;
  ua.Wc = wc;
  if (!hh::uq_general_scratch(wr, wc)) return;
  ua.gscr_stride = hh::uq_general_stride(wr, wc);
  ua.gscr_slices = 4 * ctx->num_sms;
}
inline hh_status uq_prepare(hh_ctx* ctx, int wr, int wc, hh::UQArgs& ua) {
  uq_setup(ctx, wr, wc, ua);
  if (!hh::uq_general_scratch(wr, wc)) return HH_OK;
  return buf(ctx, "uq_scratch", (size_t)ua.gscr_slices * ua.gscr_stride, &ua.gscr);
}

// Launch the correlation of one pass: the fused kernel where one exists,
// else the general-shape kernel (gcorr_prepare must have filled ca).
inline cudaError_t corr_launch(hh_ctx* ctx, const hh_pass_desc& p, const CorrArgs& ca, cudaStream_t s) {
  if (corr_special(p)) return hh::launch_correlate(ca, fft_size(p), p.search[0], s, ctx->num_sms);
  return hh::launch_correlate_general(ca, s);
}

inline hh_status set_device(hh_ctx* ctx) {
  HH_CK(cudaSetDevice(ctx->device));
  return HH_OK;
}

// B-spline elimination factors of one line length, built once per context.
inline hh_status bs_factors(hh_ctx* ctx, int64_t n, float** cp, float** inv) {
  auto it = ctx->bs_factors.find(n);
  if (it == ctx->bs_factors.end()) {
    float *a = nullptr, *b = nullptr;
    HH_CK(cudaMalloc(&a, std::max<int64_t>(n, 1) * sizeof(float)));
    HH_CK(cudaMalloc(&b, std::max<int64_t>(n, 1) * sizeof(float)));
    HH_CK(hh::launch_bspline_factors(n, a, b, ctx->stream));
    ctx->launches += 1;
    it = ctx->bs_factors.emplace(n, std::make_pair(a, b)).first;
  }
  *cp = it->second.first;
  *inv = it->second.second;
  return HH_OK;
}

inline cudaEvent_t pool_event(hh_ctx* ctx) {
  if (!ctx->evpool.empty()) {
    cudaEvent_t e = ctx->evpool.back();
    ctx->evpool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

// Launch one or more kernels of class cls; count them, and when profiling
// bracket them with events on the context stream.
template <class F>
inline hh_status run_k(hh_ctx* ctx, int cls, int nk, double flops, double bytes, int64_t units, F&& f) {
  cudaEvent_t a = nullptr;
  if (ctx->prof) {
    a = pool_event(ctx);
    cudaEventRecord(a, ctx->stream);
  }
  cudaError_t e = f();
  if (e != cudaSuccess)
    return fail(ctx, e == cudaErrorMemoryAllocation ? HH_ERR_OOM : HH_ERR_CUDA,
                std::string("kernel launch failed: ") + cudaGetErrorString(e));
  ctx->launches += nk;
  if (ctx->prof) {
    cudaEvent_t b = pool_event(ctx);
    cudaEventRecord(b, ctx->stream);
    ctx->pending.push_back({cls, a, b, flops, bytes, units, nk});
  }
  return HH_OK;
}
#define HH_K(cls, nk, fl, by, un, call) HH_TRY(run_k(ctx, cls, nk, (double)(fl), (double)(by), (int64_t)(un), [&]() { return (call); }))

// Fold completed event pairs into the per-class totals (stream synchronised).
inline hh_status flush_profile(hh_ctx* ctx) {
  for (auto& q : ctx->pending) {
    float ms = 0.f;
    HH_CK(cudaEventElapsedTime(&ms, q.a, q.b));
    hh_kernel_profile& t = ctx->acc[q.cls];
    t.launches += q.nk;
    t.ms += ms;
    t.flops += q.flops;
    t.bytes += q.bytes;
    t.units += q.units;
    ctx->evpool.push_back(q.a);
    ctx->evpool.push_back(q.b);
  }
  ctx->pending.clear();
  return HH_OK;
}

// algorithmic work of one correlation launch: 2 forward + 1 inverse real
// 2-D FFT (2.5 M log2 M each, M = N^2) + 8 M for spectrum and gain per
// window; bytes: both windows read once, packed scalars written.
inline double corr_flops(int N, int64_t njobs) {
  const double M = (double)N * N;
  return (double)njobs * (3.0 * 2.5 * M * std::log2(M) + 8.0 * M);
}
inline double corr_bytes(int W, int nalt, int64_t njobs) { return (double)njobs * (2.0 * W * W * 4 + 4.0 * (4 + 2 * nalt)); }
// the same for a pass of any shape: FFT plane NR x NC, frame-A window and
// frame-B search area read once
inline double corr_flops(const hh_pass_desc& p, int64_t njobs) {
  const double M = (double)fft_rows(p) * fft_cols(p);
  return (double)njobs * (3.0 * 2.5 * M * std::log2(M) + 8.0 * M);
}
inline double corr_bytes(const hh_pass_desc& p, int nalt, int64_t njobs) {
  return (double)njobs * (4.0 * ((double)p.window[0] * p.window[1] + (double)p.search[0] * p.search[1]) +
                          4.0 * (4 + 2 * nalt));
}
inline double uq_flops(int W, int64_t njobs) { return (double)njobs * 2.0 * 2.0 * (3 + 41) * W * (W - 1); }
inline double uq_flops(const hh_pass_desc& p, int64_t njobs) {
  const double wr = p.window[0], wc = p.window[1];
  return (double)njobs * 2.0 * (3 + 41) * (wr * (wc - 1) + wc * (wr - 1));
}

// Cubic B-spline coefficients of both images of a pair.
inline hh_status prefilter_pair(hh_ctx* ctx, const float* dA, const float* dB, int64_t nr, int64_t nc, float* cA, float* cB) {
  float *cpc, *ivc, *cpr, *ivr, *bsd;
  HH_TRY(bs_factors(ctx, nr + 2, &cpc, &ivc));
  HH_TRY(bs_factors(ctx, nc + 2, &cpr, &ivr));
  HH_TRY(buf(ctx, "bs_dbuf", (size_t)2 * (nr + 2) * (nc + 2), &bsd));
  const double P = (double)nr * nc;
  HH_K(HH_K_PREFILTER, 4, 24 * P, 16 * P, (int64_t)(2 * P),
       hh::launch_prefilter_pair(dA, dB, nr, nc, cA, cB, bsd, cpc, ivc, cpr, ivr, ctx->stream));
  return HH_OK;
}


// validate_and_replace! (src/pipeline.jl:617-645) on device buffers.
inline hh_status validate_device(hh_ctx* ctx, const hh_pass_desc& p, int ny, int nx, float* u, float* v, const float* ratio,
                          const float* moment, uint8_t* outl, uint8_t* outl2, const uint8_t* gmask, bool any_mask,
                          const float* alt_u, const float* alt_v, int nalt, bool force_replace) {
  cudaStream_t s = ctx->stream;
  const int64_t G = (int64_t)ny * nx;
  const uint8_t* gm = any_mask ? gmask : nullptr;
  hh::FlagRules r{p.uod_enable, p.uod_neighborhood, p.uod_threshold, p.min_peak_ratio, p.n_validators};
  std::copy(p.validators, p.validators + p.n_validators, r.val);
  const bool subst = alt_u && nalt > 0;
  HH_K(HH_K_VECTOR, 1, 0, 48 * G, G, hh::launch_flags(u, v, ratio, moment, ny, nx, r, gm, outl, subst ? outl2 : nullptr, s));
  if (subst)
    HH_K(HH_K_VECTOR, 1, 0, (10 + 8 * nalt) * G, G,
         hh::launch_substitute(u, v, outl2, outl, gm, alt_u, alt_v, nalt, ny, nx, p.uod_neighborhood, p.uod_threshold, s));
  if (force_replace || p.replace_outliers)
    HH_K(HH_K_VECTOR, 1, 0, 10 * G, G, hh::launch_replace(u, v, outl, gm, ny, nx, 1, s));
  return HH_OK;
}

// The grids of every pass and, with an image mask on the device, their grid
// masks and window lists: counted on the device, one copy back for all passes.
inline hh_status pass_grids(hh_ctx* ctx, int64_t nr, int64_t nc, const hh_pass_desc* passes, int np, const uint8_t* dmask,
                            double thr, std::vector<Grid>& grids) {
  grids.assign(np, Grid());
  int64_t tot = 0;
  for (int k = 0; k < np; ++k) {
    HH_TRY(grid_axes(ctx, nr, nc, passes[k], grids[k]));
    tot += grids[k].G();
  }
  if (!dmask) return HH_OK;
  uint8_t* d;
  HH_TRY(buf(ctx, "gmask_all", tot, &d));
  int64_t off = 0;
  for (int k = 0; k < np; ++k) {
    const hh_pass_desc& p = passes[k];
    const Grid& g = grids[k];
    HH_K(HH_K_VECTOR, 1, 0, g.G(), g.G(),
         hh::launch_mask_grid(dmask, nr, g.ny, g.nx, g.win, p.window[0], p.window[1], (p.search[0] - p.window[0]) / 2,
                              (p.search[1] - p.window[1]) / 2, thr, d + off, ctx->stream));
    off += g.G();
  }
  std::vector<uint8_t> h(tot);
  HH_CK(cudaMemcpyAsync(h.data(), d, tot, cudaMemcpyDeviceToHost, ctx->stream));
  HH_CK(cudaStreamSynchronize(ctx->stream));
  off = 0;
  for (Grid& g : grids) {
    g.gmask.assign(h.begin() + off, h.begin() + off + g.G());
    g.any_mask = std::any_of(g.gmask.begin(), g.gmask.end(), [](uint8_t m) { return m != 0; });
    if (g.any_mask) grid_jobs(g);
    off += g.G();
  }
  return HH_OK;
}
// windows of a grid from pass_grids
inline int64_t grid_njobs(const Grid& g) { return g.any_mask ? (int64_t)g.jobs.size() / 4 : g.G(); }
// its window list and grid mask on the device (the mask only where a cell is masked)
inline hh_status stage_grid(hh_ctx* ctx, const Grid& g, int32_t* djobs, uint8_t* gm) {
  cudaStream_t s = ctx->stream;
  if (!g.any_mask) {
    HH_K(HH_K_VECTOR, 1, 0, 16 * g.G(), g.G(), hh::launch_make_jobs(djobs, g.ny, g.nx, g.win, s));
    return HH_OK;
  }
  HH_CK(cudaMemcpyAsync(djobs, g.jobs.data(), g.jobs.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  HH_CK(cudaMemcpyAsync(gm, g.gmask.data(), g.G(), cudaMemcpyHostToDevice, s));
  return HH_OK;
}
// predictor nodes of grid g
inline hh::PredGrid pred_grid(const Grid& g) {
  return hh::PredGrid{g.ny, g.nx, g.y[0], g.ny > 1 ? g.y[1] - g.y[0] : 1.f, g.x[0], g.nx > 1 ? g.x[1] - g.x[0] : 1.f};
}
// predictor (u, v) on nodes pg, wanted on grid g
inline hh::NodePred node_pred(const float* u, const float* v, const hh::PredGrid& pg, const Grid& g) {
  const hh::PredGrid n = pred_grid(g);
  return hh::NodePred{u, v, pg, n.y0, n.ysp, n.x0, n.xsp};
}

// Device storage of the final fields as one block of G cells per field, in
// the order u, v, ratio, moment, flags (a byte each), uncertainties: a result
// that fits the context's page-locked block comes back in one copy.
struct ResultBlock {
  float *u, *v, *ratio, *moment, *uncu, *uncv;
  uint8_t* outl;
};
inline hh_status result_block(hh_ctx* ctx, int64_t G, ResultBlock& r) {
  const int64_t fw = (G + 3) / 4;  // words of the flags
  HH_TRY(buf(ctx, "result", (size_t)(6 * G + fw), &r.u));
  r.v = r.u + G;
  r.ratio = r.v + G;
  r.moment = r.ratio + G;
  r.outl = reinterpret_cast<uint8_t*>(r.moment + G);
  r.uncu = r.moment + G + fw;
  r.uncv = r.uncu + G;
  return HH_OK;
}
// G: cells the block was laid out for; unc: whether uncertainties were estimated (else they are NaN)
inline hh_status read_results(hh_ctx* ctx, const Grid& g, const ResultBlock& r, int64_t Gb, bool unc, hh_result* out) {
  cudaStream_t s = ctx->stream;
  const int64_t G = g.G();
  out->ny = g.ny;
  out->nx = g.nx;
  if (out->x) memcpy(out->x, g.x.data(), g.nx * sizeof(float));
  if (out->y) memcpy(out->y, g.y.data(), g.ny * sizeof(float));
  struct Field {
    void* dst;
    const void* src;
    size_t bytes;
  } f[7] = {{out->u, r.u, G * sizeof(float)},
            {out->v, r.v, G * sizeof(float)},
            {out->peak_ratio, r.ratio, G * sizeof(float)},
            {out->correlation_moment, r.moment, G * sizeof(float)},
            {out->outliers, r.outl, (size_t)G},
            {unc ? out->uncertainty_u : nullptr, r.uncu, G * sizeof(float)},
            {unc ? out->uncertainty_v : nullptr, r.uncv, G * sizeof(float)}};
  const char* base = reinterpret_cast<const char*>(r.u);
  const size_t total = (unc ? 6 * Gb + (Gb + 3) / 4 : 4 * Gb + (Gb + 3) / 4) * sizeof(float);
  if (total <= HH_PINNED_BYTES) {
    HH_CK(cudaMemcpyAsync(ctx->pinned, base, total, cudaMemcpyDeviceToHost, s));
    HH_CK(cudaStreamSynchronize(s));
    const char* h = reinterpret_cast<const char*>(ctx->pinned);
    for (const Field& q : f)
      if (q.dst) memcpy(q.dst, h + (static_cast<const char*>(q.src) - base), q.bytes);
  } else {
    for (const Field& q : f)
      if (q.dst) HH_CK(cudaMemcpyAsync(q.dst, q.src, q.bytes, cudaMemcpyDeviceToHost, s));
    HH_CK(cudaStreamSynchronize(s));
  }
  if (!unc)
    for (float* q : {out->uncertainty_u, out->uncertainty_v})
      if (q) std::fill(q, q + G, std::nanf(""));
  if (out->mask) {
    if (g.any_mask) memcpy(out->mask, g.gmask.data(), G);
    else memset(out->mask, 0, G);
  }
  return HH_OK;
}

inline hh_status read_scalar(hh_ctx* ctx, const float* dptr, float* out) {
  HH_CK(cudaMemcpyAsync(ctx->pinned, dptr, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  HH_CK(cudaStreamSynchronize(ctx->stream));
  *out = ctx->pinned[0];
  return HH_OK;
}

inline hh_status check_passes(hh_ctx* ctx, const hh_pass_desc* passes, int np) {
  if (!passes || np < 1) return fail(ctx, HH_ERR_ARG, "at least one pass is required");
  for (int k = 0; k < np; ++k) {
    hh_status s = hh_pass_validate(&passes[k]);
    if (s != HH_OK) return fail(ctx, s, hh_last_error(nullptr));
  }
  hh_status s = hh_check_backend_params(passes, np);
  if (s != HH_OK) return fail(ctx, s, hh_last_error(nullptr));
  return HH_OK;
}


}  // namespace hhd
