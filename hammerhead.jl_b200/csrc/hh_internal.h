// Internal declarations shared by the C-ABI layer and the kernel files.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>

#include "hammerhead_b200.h"

namespace hh {

struct BPair;

constexpr int KMAX = 8;  // peaks tracked per window on the device (n_peaks <= 8)

// B-spline prefilter: each line's two Thomas sweeps are cut into independent
// segments of BS_SEG unknowns whose sweeps start BS_WARM unknowns early from a
// zero state (k_deform.cu). Segments of a padded line of n elements (n - 4
// unknowns); the batched plan counts its work items with it.
constexpr int BS_SEG = 64, BS_WARM = 32;
__host__ __device__ __forceinline__ int64_t b_nseg(int64_t n) { return n >= 5 ? (n - 4 + BS_SEG - 1) / BS_SEG : 1; }

// Arguments of the fused correlation kernel (one pass, one image pair).
struct CorrArgs {
  const float* A;            // deformed (or raw) frame A, column-major nr x nc
  const float* B;            // frame B
  const uint8_t* mask;       // image mask (nonzero = excluded) or nullptr
  int64_t ld;                // leading dimension (= nr)
  const int32_t* jobs;       // 4 int32 per job: gi, gj, rs, cs (0-based)
  int64_t njobs;
  int32_t ny;                // grid rows; grid index id = gi + gj * ny
  int64_t G;                 // grid size ny * nx
  const float* apod;         // W x W apodization window (column-major)
  const float* gain;         // N x N overlap gain (fftshifted layout) or nullptr
  const float* phasew;       // N x N phase filter (natural FFT order) or nullptr
  int32_t method, npeaks, finder, subpixel;
  // grid-indexed outputs (residual displacement of this sweep)
  float* du;
  float* dv;
  float* ratio;
  float* moment;
  float* alt_u;              // G x nalt or nullptr
  float* alt_v;
  int32_t nalt;
  // optional per-job outputs
  float* packed;             // (5 + 2(K-1)) x njobs
  int32_t* locs;             // 2K x njobs (1-based row, col)
  float* planes;             // N*N x njobs correlation planes
  // batched mode (bp != nullptr): jobs are (pair, gi | gj << 16, rs, cs);
  // images, grid offsets and sizes come from bp[pair]; windows of pairs not
  // live in sweep `it` are skipped
  const BPair* bp;
  const int32_t* done;
  int32_t it;
  // ensemble mode: planes += R (planes != nullptr) and no peak analysis
  int32_t accumulate;
  // fftshifted rows/columns [box_lo, box_hi] outside which the overlap gain
  // is zero (box_hi == 0: the whole plane); with an enlarged search area the
  // lags kept by restrict_search_lags! (src/correlators.jl:347-355)
  int32_t box_lo, box_hi;
  // enlarged search area: the launch's W is the frame-B search area and win
  // the frame-A window centred in it (jobs give the window's origin); 0 when
  // the two are equal
  int32_t win;
  // CTA shape of the launch (0: default, 1: the alternative; equal areas only)
  int32_t variant;
  // peak records (correlate_record_words(npeaks) x njobs floats) or nullptr:
  // with regional maxima the per-window outputs are then formed by a
  // one-thread-per-window epilogue kernel after the correlation kernel
  float* rec;
  // general-shape path (correlate_general_kernel): window wr x wc, search
  // area sr x sc, FFT plane nfr x nfc; gscr holds one scratch slice of
  // gscr_stride float2 per CTA (complex and real plane; none when they live in
  // shared memory), gscr_slices is the number of CTAs; twr / twc the
  // twiddle tables exp(-2 pi i t / n) of the two lengths and their radix
  // plans; the line buffers' layout and shared bytes
  int32_t wr, wc, sr, sc, nfr, nfc;
  float2* gscr;
  int64_t gscr_stride;
  int32_t gscr_slices;
  const float2* twr;
  const float2* twc;
  int8_t gc_radix_r[24], gc_radix_c[24];
  int32_t gc_nst_r, gc_nst_c;
  int32_t gc_col_warps, gc_chunk_c;  // warps of the columns passes (one line each); rows-pass lines per chunk
  int64_t gc_smem_lines;
  int32_t gc_threads, gc_in_smem;  // threads per CTA; whether the planes live in shared memory
  int64_t gc_smem_bytes;           // shared memory per CTA
  // fftshifted rows [0], [1] and columns [2], [3] outside which the plane is
  // zero (overlap-gain support or kept search lags; the whole plane otherwise)
  int32_t gc_box[4];
};

// Launch the correlation kernel for FFT size N (square) and window W (the
// search area when a.win is set).
cudaError_t launch_correlate(const CorrArgs& a, int N, int W, cudaStream_t s, int num_sms);
// outputs from the peak records of a fused correlation launch of FFT size N
cudaError_t launch_peak_epilogue(const CorrArgs& a, int N, cudaStream_t s, int num_sms);
bool correlate_supported(int N, int W);
// The general-shape correlation (any FFT lengths, rectangular windows and
// search areas): a.wr .. a.gc_smem_lines set by the host (gcorr_prepare).
cudaError_t launch_correlate_general(const CorrArgs& a, cudaStream_t s);
// shared memory of a general-shape CTA beside its line buffers and planes
__host__ __device__ constexpr size_t gcorr_smem_extra(int warps) {
  return warps * (4 * sizeof(double) + 2 * KMAX * sizeof(uint32_t)) + KMAX * (sizeof(float) + 2 * sizeof(int)) + 64;
}
// CTAs of 128 threads per SM of the kernel that holds the planes in shared
// memory (hh_corr_plane.cuh), and its shared memory per CTA
constexpr int gcorr_plane_ctas = 6;
size_t gcorr_plane_smem(int nr, int nc, int box_rows, int box_cols, int threads);
// Radix plan of an FFT length (factors 4, 2, then odd primes <= 61);
// returns the stage count, or -1 when a factor exceeds 61 or there are more
// than 24 stages.
int gcorr_radix_plan(int n, int8_t* radix);
size_t correlate_record_words(int npeaks);  // per job

// Device peak analysis of caller-supplied planes.
struct AnalyzeArgs {
  const float* planes;
  int64_t nplanes;
  int32_t nr, nc;
  int32_t npeaks, finder, subpixel;
  float* packed;
  int32_t* locs;
  // optional grid outputs (as CorrArgs): plane j is job j of `jobs`
  const int32_t* jobs;
  int32_t ny;
  int64_t G;
  float *du, *dv, *ratio, *moment, *alt_u, *alt_v;
  int32_t nalt;
};
cudaError_t launch_analyze_planes(const AnalyzeArgs& a, cudaStream_t s);

// --- deformation -----------------------------------------------------------
cudaError_t launch_bspline_factors(int64_t n, float* cp, float* inv, cudaStream_t s);
// Cubic B-spline coefficients ((nr + 2) x (nc + 2), padded) of both frames of
// a pair; dbuf: 2 (nr + 2) (nc + 2) floats for the forward sweeps.
cudaError_t launch_prefilter_pair(const float* imgA, const float* imgB, int64_t nr, int64_t nc, float* coefA,
                                  float* coefB, float* dbuf, const float* cpc, const float* ivc, const float* cpr,
                                  const float* ivr, cudaStream_t s);
struct PredGrid {
  int32_t gny, gnx;
  float y0, ysp, x0, xsp;
};
// a deformation's form for images of nr rows, its warps' work items in strips of
// `cols` columns, and how many columns a launch takes whose strips they give
bool deform_wraps(int64_t nr);
int64_t deform_strips(bool wrap, int64_t nr, int64_t nc, int cols);
int deform_cols(const std::function<int64_t(int)>& strips);
cudaError_t launch_deform(const float* CA, const float* CB, int64_t nr, int64_t nc, const float* pu,
                          const float* pv, PredGrid g, float* wA, float* wB, cudaStream_t s);
cudaError_t launch_node_values(const float* pu, const float* pv, PredGrid g, const float* y, int32_t ny,
                               const float* x, int32_t nx, float* u, float* v, cudaStream_t s);

// --- vector-grid kernels -----------------------------------------------------
// a predictor on nodes (u, v) and the grid it is wanted on: node (gi, gj) at
// (y0 + gi ysp, x0 + gj xsp); u == nullptr: no predictor
struct NodePred {
  const float* u;
  const float* v;
  PredGrid g;
  float y0, ysp, x0, xsp;
};
// validation rules of a pass (hh_pass_desc)
struct FlagRules {
  int32_t uod, uod_nb;
  double uod_thr, min_ratio;
  int32_t nval;
  hh_validator val[HH_MAX_VALIDATORS];
};
// the windows of a grid: 0-based first pixel of window (gi, gj) at
// (r0 + gi rstep, c0 + gj cstep)
struct WinGrid {
  int32_t r0, rstep, c0, cstep;
};
cudaError_t launch_combine(float* u, float* v, const float* resu, const float* resv, float* ratio, float* moment,
                           float* alt_u, float* alt_v, int32_t nalt, const uint8_t* gmask, int32_t ny, int32_t nx,
                           const NodePred& pr, float* meas_u, float* meas_v, cudaStream_t s);
cudaError_t launch_flags(const float* u, const float* v, const float* ratio, const float* moment, int32_t ny, int32_t nx,
                         const FlagRules& r, const uint8_t* gmask, uint8_t* flags, uint8_t* flags2, cudaStream_t s);
// kernels that launch_predictor launches: the fill, and the smoothing or the copy of the field
constexpr int predictor_launches(bool masked, bool smoothing, bool keep) {
  return (masked || !smoothing) + (smoothing || keep);
}
cudaError_t launch_predictor(const float* u, const float* v, const uint8_t* gmask, int32_t ny, int32_t nx, bool smoothing,
                             float* wu, float* wv, float* ou, float* ov, float* prev_u, float* prev_v, cudaStream_t s);
cudaError_t launch_make_jobs(int32_t* jobs, int32_t ny, int32_t nx, const WinGrid& w, cudaStream_t s);
cudaError_t launch_mask_grid(const uint8_t* mask, int64_t nr, int32_t ny, int32_t nx, const WinGrid& w, int32_t wr,
                             int32_t wc, int32_t mr, int32_t mc, double thr, uint8_t* gmask, cudaStream_t s);
cudaError_t launch_uod(const float* u, const float* v, int32_t ny, int32_t nx, double thr, int32_t nb, double eps,
                       const uint8_t* exclude, uint8_t* flags, int32_t or_into, cudaStream_t s);
cudaError_t launch_substitute(float* u, float* v, const uint8_t* outl_in, uint8_t* outl_out, const uint8_t* gmask,
                              const float* alt_u, const float* alt_v, int32_t nalt, int32_t ny, int32_t nx,
                              int32_t er, double thr, cudaStream_t s);
// replace_vectors!: invalid = flags | gmask (either may be nullptr); masked
// cells are set to NaN afterwards when nan_mask is nonzero.
cudaError_t launch_replace(float* u, float* v, const uint8_t* flags, const uint8_t* gmask, int32_t ny, int32_t nx,
                           int32_t nan_mask, cudaStream_t s);
cudaError_t launch_smooth(const float* f, int32_t ny, int32_t nx, float* out, cudaStream_t s);
// field_change -> *out (device float); scratch: G floats + 2 KB
cudaError_t launch_field_change(const float* u, const float* v, const float* pu, const float* pv,
                                const uint8_t* gmask, int64_t G, float* scratch, float* out, cudaStream_t s);
cudaError_t launch_restore_measured(float* u, float* v, const float* meas_u, const float* meas_v,
                                    const uint8_t* outl, int64_t G, cudaStream_t s);
cudaError_t launch_fill(float* p, float value, int64_t n, cudaStream_t s);

// --- ingestion -------------------------------------------------------------------
// UInt16 frame -> float32: value / 65535 (normalise) or value * 1
cudaError_t launch_u16_to_f32(const uint16_t* src, int64_t n, int32_t normalise, float* dst, cudaStream_t s);

// --- uncertainty -------------------------------------------------------------
struct UQArgs {
  const float* A;
  const float* B;
  const uint8_t* mask;
  int64_t ld;
  const int32_t* jobs;
  int64_t njobs;
  int32_t ny;
  int32_t W;
  const float* apod;
  double* stats;     // 88 per job, or nullptr
  float* unc_u;      // grid-indexed outputs, or nullptr
  float* unc_v;
  // batched mode (bp != nullptr): jobs as in CorrArgs; mode 0 = the fused
  // estimate of a single-sweep pass (sweep 1), 1 = the post-loop estimate
  const BPair* bp;
  const int32_t* done;
  int32_t mode;
  // ensemble mode: stats += this pair's statistics
  int32_t accumulate;
  // rectangular windows (W rows x Wc columns; Wc == 0: square) and windows
  // above 64 px run the general form, whose per-window buffers live in a
  // global scratch slice per CTA (gscr_slices slices of gscr_stride doubles)
  int32_t Wc;
  double* gscr;
  int64_t gscr_stride;
  int32_t gscr_slices;
};
cudaError_t launch_uq(const UQArgs& a, cudaStream_t s, int num_sms);
// Does this window shape run the general (global-scratch) form, and how many
// doubles does one window's scratch slice take?
bool uq_general(int wr, int wc);
bool uq_general_scratch(int wr, int wc);  // ... and does it need the scratch (else shared memory)?
int64_t uq_general_stride(int wr, int wc);
// finalize_uncertainty of pooled statistics (88 per job) into grid cells
cudaError_t launch_uq_finalize(const double* stats, const int32_t* jobs, int64_t njobs, int32_t ny, float* unc_u,
                               float* unc_v, cudaStream_t s);

// --- adjoint of deformation + zero-lag correlation --------------------------
struct NccArgs {
  const float* CA;  // B-spline coefficients of both frames, (nr + 2) x (nc + 2)
  const float* CB;
  int64_t nr, nc;
  const float* P;   // predictor: u plane then v plane, gny x gnx each
  int32_t gny, gnx;
  float y0, ysp, x0, xsp;
  int32_t W, step;  // windows: W x W at origins (jr * step, jc * step)
  int32_t wy, wx;   // window grid
  double* wstat;    // ncc_wstat_words (scratch): 6 per window, then a sum per tile of windows
  float* gpix;      // 2 x nr x nc pixel gradient (scratch), when grad
  int32_t* cells;   // predictor cell and fraction bits per row, then per column (scratch), when grad
  float* grad;      // 2 x gny x gnx dL/dP, or nullptr (loss only)
  double* loss;     // device scalar
};
int64_t ncc_wstat_words(int32_t wy, int32_t wx);
cudaError_t launch_ncc_loss_grad(const NccArgs& a, cudaStream_t s);

}  // namespace hh
