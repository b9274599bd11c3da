// Fused window correlation for the planar WIDIM pass (sm_100a).
//
// One CTA holds WPC interrogation windows in shared memory and runs, per
// window, the whole of the reference's per-window chain
//   load_windows!  (src/correlators.jl:188-263: column-major mean, apodize)
//   FFT A, FFT B   (packed as one complex transform of A + iB)
//   spectrum!      (src/correlators.jl:266-279: conj(FA) FB, or filtered phase)
//   inverse FFT    (normalised by 1/N^2 like FFTW's inv(plan))
//   fftshift_abs!, overlap gain (src/correlators.jl:282-289, 338-339)
//   analyze_plane! (src/correlators.jl:459-468: regional-max or exclusion
//                   peaks with the tie rules of src/localmax.jl:3-19,
//                   gauss3/gauss9 in FP64, peak ratio, FP64 moment,
//                   gauss3-refined alternatives)
// writing the packed scalars of src/ka_backend.jl:497-506 straight into the
// vector grid. Nothing but images in and scalars out touches HBM.
//
// Shared-memory plane layout: element (p, q) (row p, column q) of window w
// lives at planes[w*N*LD + q*LD + p] with LD = N + 1, so a warp walking
// either axis with one line per lane is bank-conflict free.
//
// The 2-D transform runs each axis as an in-register radix-N1 pass and, for
// N > 32, a second radix-N2 pass (N = N1*N2). The forward transform leaves
// frequency k at position N2*(k % N1) + k / N1 along each axis; the spectrum
// is formed from pairs (k, -k) there and the inverse takes that order back
// to natural order, so no bit-reversal pass exists anywhere.
#pragma once
#include "hh_attr.h"
#include "hh_corr_peaks.cuh"
#include "hh_corr_seg.cuh"

namespace hh {

// ---------------------------------------------------------------------------
// W is the extent of the data: the window, or with SRCH the frame-B search
// area that holds the (runtime) frame-A window at its centre. VAR selects the
// CTA shape (windows per CTA, threads per window) and register budget (CTAs
// per SM the registers are sized for) and FFT split among the five the
// autotuner times: 0 the default shape and budget, 1 the alternative shape,
// 2 the default shape with one CTA per SM more in the budget (fewer
// registers, more warps), 3 the default shape with one CTA less (more
// registers, no spills) -- or, where the default budget is one CTA, the
// alternative shape with one CTA more. Variants 0-3 compute the same
// arithmetic on another thread mapping or register allocation, so their
// results are identical. Variant 4 splits each axis's DFT differently
// (AxisSplitAlt), so its planes differ from variant 0's by rounding. (At 16
// and 32 points a launch of variant 0 with enough windows takes another kernel
// with the same arithmetic: launch_corr_nw.)
template <int N, int W, bool SRCH = false, int VAR = 0> struct CorrCfg {
  // variant 4: the alternative FFT split (AxisSplitAlt) in the default shape and budget
  static constexpr bool ALT = VAR == 4;
  static constexpr int N1 = ALT ? AxisSplitAlt<N>::N1 : AxisSplit<N>::N1;
  static constexpr int N2 = ALT ? AxisSplitAlt<N>::N2 : AxisSplit<N>::N2;
  // budget of the default shape; shape of this variant (0 default, 1 alternative)
  static constexpr int MINB0 = (N == 32 && W == 16) ? 3 : (N <= 48 ? 4 : (N <= 64 ? 3 : (N <= 96 ? 2 : 1)));
  static constexpr int SH = (VAR == 1 || (VAR == 3 && MINB0 == 1)) ? 1 : 0;
  // 16 x 16 windows padded to 32: every stage of the plane has at most 16
  // lines (16 data columns, 16 canonical column items, 16 row pairs), so
  // half a warp serves a window and each warp carries two
  static constexpr bool HALF = SH == 0 && N == 32 && W == 16;
  // alternatives: N <= 32 one window per warp in CTAs of 4 (half-warp
  // windows) or 8 warps; N = 48 a 3-CTA register budget; N = 64 one window
  // per 256-thread CTA; N = 96 512 threads and N = 128 256 threads per window
  static constexpr int WPC = SH == 0 ? (HALF ? 8 : (N <= 32 ? 4 : (N <= 64 ? 2 : 1)))  // windows per CTA
                                     : (N <= 32 ? (N == 32 && W == 16 ? 4 : 8) : (N <= 48 ? 2 : 1));
  static constexpr int NT = SH == 0 ? (N <= 48 ? 128 : (N <= 96 ? 256 : 512))
                                    : (N <= 32 ? (N == 32 && W == 16 ? 128 : 256)
                                               : (N <= 48 ? 128 : (N <= 64 ? 256 : (N <= 96 ? 512 : 256))));
  static constexpr int G = NT / WPC;  // threads per window
  // CTAs per SM the register budget is sized for
  static constexpr int MINB_SH = SH == 0 ? MINB0
                                         : (N <= 32 ? (N == 32 && W == 16 ? 4 : 2) : (N <= 48 ? 3 : (N <= 64 ? 3 : 1)));
  static constexpr int MINB = VAR == 2 ? MINB0 + 1
                                       : (VAR == 3 ? (MINB0 > 1 ? MINB0 - 1 : MINB_SH + 1) : MINB_SH);
  // the peak analysis inline (one window per CTA: its latency is the CTA's)
  static constexpr bool INLINE_ANALYSIS = N >= 96;
  // Canonical column c = N1 u + v sits at storage column N2 v + u, and with
  // LD = N + 1 a 64-bit element's bank pair is (column + row) mod 16: row slot
  // N2 k1 + k2 of the first inverse pass along p falls on N2 (v + k1) + u + k2.
  // Consecutive canonical columns share two (N2 = 8) or four (N2 = 4) bank
  // pairs; with u fastest, half a warp covers u < N2/2 and 32 / N2 values of v,
  // still two to a bank pair, since every term but u is a multiple of N2 or
  // common. So every other run of 16 / N2 values of v swaps the halves of its
  // groups: it takes slot k2 ^ N2/2 for k2, which turns the sign of the odd
  // outputs (turned back in the twiddle) and leaves row N2 n1 + n2 of those
  // columns at row slot N2 n1 + (n2 ^ N2/2), where the last axis looks for it
  // (rot). For N2 = 6 the columns of u = 0 and 1 cover the bank pairs with v
  // fastest, and those of u = 2 half of them. A model of the
  // pass's addresses gives 1152 wavefronts at 128 points (ideal 1040, without
  // the swap 2176), 672 at 96 (588; 1248), 288 at 64 (264; 880 in column
  // order), 204 at 48 (150; 288 in column order).
  static constexpr bool ROT = N2 == 4 || N2 == 8;
  static __host__ __device__ constexpr int rot(int v) { return ROT ? (v / (16 / N2) & 1) * (N2 / 2) : 0; }
  // The spectrum is Hermitian, so the inverse transforms only the N/2 + 1
  // canonical columns along p and then rows p and p + N/2 together along q
  // (their outputs are real: one lands in the real part, one in the
  // imaginary part). Every window is transformed on its own.
  static constexpr int NC = N / 2 + 1;
  static constexpr int LD = N + 1;    // complex plane leading dimension (float2)
  static constexpr int LDR = N + 1;   // real plane leading dimension (float), overlays the complex plane
  static constexpr bool PADDED = (W * 2 == N);
  // A padded window keeps only lags |lag| <= N/4 on either axis: the overlap
  // gain is zero where the weight (the apodization window's autocorrelation)
  // is below half its maximum, which for the triangle of the plain window
  // starts past W/2 = N/4 and for the Gaussian earlier (6 of 32 points). So
  // both inverse axes form only the outputs that hold such a lag: keep(n1)
  // of the last pass (the others' butterflies fold away and nothing is
  // stored for them), at most Q + 1 row pairs, and a real plane whose cells
  // outside the box are never stored but read as the zeros they are. Half of
  // the inverse's stores and a third of its arithmetic are for lags outside
  // N/4. launch_nw checks that the table's box is inside it.
  static constexpr bool BOXED = PADDED && !SRCH;
  static constexpr int Q = N / 4;
  static constexpr bool keep(int n1) { return !BOXED || N2 * n1 <= Q || N2 * n1 + N2 - 1 >= N - Q; }
  static constexpr int NHMAX = BOXED ? Q + 1 : N / 2;  // row pairs of the last inverse axis
  static constexpr int IPT = (NHMAX * N2 + G - 1) / G;  // final inverse items per thread
  static constexpr int NZ1 = PADDED ? (W / N2) : N1;  // nonzero inputs of a forward pass-A line

  static constexpr int EPT = (W * W + G - 1) / G;             // window pixels per thread
  // pixels wait in the plane for their mean, not in registers, where they would
  // spill: search areas of 96 px 558 -> 446 us for 2500 windows, 64 px 166 -> 132,
  // 48 px (phase) 228 -> 168; the 18 pixels of a 24 px area do better in registers
  static constexpr bool VIA = EPT > (SRCH ? 18 : 16);
  static constexpr int NPART = SRCH ? 4 : 3;  // FP64 partial sums per warp: A, B, count (and count of B)
  // plane stride in float2; the two windows of a half-warp pair start 16
  // banks apart, so their 32-bit plane accesses (peak scan, real-plane
  // writes) do not meet in one bank
  static constexpr int PS = N * LD + (HALF ? 8 : 0);
  static constexpr size_t PLANE_B = (size_t)PS * sizeof(float2);
  static constexpr size_t BASE_B = WPC * PLANE_B + WPC * (G / 32) * NPART * sizeof(double) + N * sizeof(float2) +
                                   WPC * (G / 32) * 2 * KMAX * sizeof(uint32_t) +
                                   WPC * (KMAX * sizeof(float) + 2 * KMAX * sizeof(int)) + N * sizeof(int) +
                                   (W == N ? WPC * N * sizeof(uint32_t) : 0) + 64;
  // The overlap gain is read by every window; from global memory its L1
  // lines are flushed by the window pixels (it took a third of the last
  // inverse pass at 32 points, half of it at 128), so the kept lags' part of
  // the table goes to shared memory. (The apodization window in shared
  // memory as well was no faster.)
  static constexpr size_t GAIN_B = BOXED ? (size_t)(2 * Q + 1) * (2 * Q + 1) * sizeof(float) : 0;
  static constexpr size_t smem() { return BASE_B + GAIN_B; }
  static_assert(W == N || 2 * W == N, "window must equal the FFT size or half of it");
  static_assert((G >= 32 && G % 32 == 0) || G == 16, "a window group is whole warps or half a warp");
  static_assert(N * LDR * 4 + (W == N ? (G + 31) / 32 * 64 * 2 : 0) <= 2 * N * LD * 4, "real plane and scan lists fit in the complex plane");
};

// ANY: the correlation method is read at run time (else cross correlation,
// without a branch per spectrum value).
template <int N, int W, bool SRCH, int VAR, bool ANY>
__global__ void __launch_bounds__(CorrCfg<N, W, SRCH, VAR>::NT, CorrCfg<N, W, SRCH, VAR>::MINB)
    correlate_kernel(const CorrArgs a) {
  using C = CorrCfg<N, W, SRCH, VAR>;
  constexpr int WPC = C::WPC, NT = C::NT, LD = C::LD, LDR = C::LDR, N1 = C::N1, N2 = C::N2, IPT = C::IPT;
  constexpr int G = C::G, EPT = C::EPT, NC = C::NC, H = N / 2;
  constexpr int PS = C::PS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* planes = reinterpret_cast<float2*>(smem_raw);
  double* s_part = reinterpret_cast<double*>(smem_raw + WPC * C::PLANE_B);  // NPART per warp
  float2* tw = reinterpret_cast<float2*>(s_part + WPC * (G / 32) * C::NPART);
  uint32_t* red = reinterpret_cast<uint32_t*>(tw + N);
  float* s_vals = reinterpret_cast<float*>(red + WPC * (G / 32) * 2 * KMAX);
  int* s_locs = reinterpret_cast<int*>(s_vals + WPC * KMAX);
  int* s_canon = s_locs + WPC * 2 * KMAX;  // storage columns of kq = 0..N/2 (N2 > 1)
  uint32_t* s_rmax = reinterpret_cast<uint32_t*>(s_canon + N);  // per window: its plane's row maxima
  float* s_gain = reinterpret_cast<float*>(s_rmax + (W == N ? WPC * N : 0));  // (2Q + 1)^2 when C::BOXED

  const int tid = threadIdx.x;
  const int method = ANY ? a.method : 0;
  const int K = a.npeaks > 2 ? a.npeaks : 2;
  constexpr int GB = 2 * C::Q + 1;
  if (C::BOXED)
    for (int m = tid; m < GB * GB; m += NT) s_gain[m] = a.gain[H - C::Q + m % GB + (H - C::Q + m / GB) * N];

  if (N2 > 1) {
    for (int m = tid; m < N; m += NT) {
      double sn, cs;
      sincospi(-2.0 * (double)m / (double)N, &sn, &cs);
      tw[m] = make_float2((float)cs, (float)sn);  // W_N^m = exp(-2 pi i m / N)
    }
    for (int q = tid; q <= N / 2; q += NT) s_canon[q] = N2 * (q % N1) + q / N1;
  }
  __syncthreads();  // the only CTA-wide barrier: from here on the window groups run independently

  // Thread group w (G threads, named barrier w + 1) owns plane w and walks
  // its own sequence of jobs; a group waits only for itself.
  const int w = tid / G, gt = tid % G, lane = tid & 31, gw = gt >> 5;
  const int bar = WPC == 1 ? 0 : w + 1;
  float2* P = planes + w * PS;
  float* Rw = reinterpret_cast<float*>(P);  // real plane, overlays the complex one after stage 8
  uint32_t* rmax = s_rmax + w * N;
  // Peak scan from the row maxima (scan_rows) where the box is the whole plane
  // or the search lags: unpadded windows. A padded window's box is at most
  // half the plane (its overlap weight halves by then) and 13 x 13 of 32 x 32
  // with the Gaussian apodization, where walking the column strips costs no
  // more (16.5 / 16.9 ns at 48 points, 28.0 / 27.6 at 64, 124 / 126 at 128)
  // and half-warp groups lose (5.6 / 10.1 ns at 32 points: the halves' loops
  // run one after the other). Unpadded, strips / row maxima: 8.8 / 7.0
  // ns at 24 points, 11.4 / 8.8 at 32, 33.6 / 26.5 at 48, 42.9 / 33.9 at 64, 154 /
  // 104 at 96, 223 / 176 at 128.
  constexpr bool ROWSCAN = W == N;
  constexpr int FN = ROWSCAN ? N : 0;
  // the peak scan's list, in the half of the plane that the real plane leaves
  uint16_t* list = reinterpret_cast<uint16_t*>(Rw + N * LDR);
  double* part = s_part + w * (G / 32) * C::NPART;
  const float scale = 1.0f / (float)(N * N);
  // fftshifted rows / columns that can hold a nonzero correlation value (the
  // support of the overlap gain; the whole plane without padding)
  const int blo = a.box_hi > 0 ? a.box_lo : 0, bhi = a.box_hi > 0 ? a.box_hi : N - 1;
  // row pairs of the last inverse axis; it / nh as a multiplication, exact for it < 1024
  const int nb = bhi - blo + 1, nh = (nb + 1) / 2;
  const uint32_t inv_nh = (65536u + nh - 1) / nh;
  const ScanPlan sp = scan_plan(tid % G, G, blo, bhi, blo, bhi);
  PeakOut po{a.du, a.dv, a.ratio, a.moment, a.alt_u, a.alt_v, a.nalt, a.G, a.packed, a.locs};

  for (int64_t job = (int64_t)blockIdx.x * WPC + w; job < a.njobs; job += (int64_t)gridDim.x * WPC) {
    // ---- the window's source (every thread of the group reads the same
    //      descriptor words; they are broadcast from L1)
    int rs, cs;
    const float* A = a.A;
    const float* B = a.B;
    const uint8_t* M = a.mask;
    int64_t ld = a.ld, gid;
    PeakOut pw = po;
    if (a.bp) {
      const int p = a.jobs[4 * job];
      const BPair& b = a.bp[p];
      const int gij = a.jobs[4 * job + 1];
      const int64_t cell = (int64_t)(gij & 0xFFFF) + (int64_t)(gij >> 16) * b.ny;
      // pairs that converged or have no further sweep, and masked cells, are skipped
      if (!bp_live(b, a.it, a.done, p) || (b.gmask && b.gmask[cell])) {
        if (a.rec && a.finder == 0 && gt == 0) a.rec[job] = __int_as_float(-1);  // no record for the epilogue
        continue;
      }
      rs = a.jobs[4 * job + 2];
      cs = a.jobs[4 * job + 3];
      const bool warped = a.it > 1 || b.has_pred0;
      A = warped ? b.warpA : b.A;
      B = warped ? b.warpB : b.B;
      M = b.mask;
      ld = b.nr;
      gid = b.goff + cell;
      pw.G = (int64_t)b.ny * b.nx;
      pw.nalt = b.nalt;
      pw.alt_u = a.alt_u ? a.alt_u + b.aoff - b.goff : nullptr;  // indexed by gid + m*G
      pw.alt_v = a.alt_v ? a.alt_v + b.aoff - b.goff : nullptr;
    } else {
      rs = a.jobs[4 * job + 2];
      cs = a.jobs[4 * job + 3];
      gid = (int64_t)a.jobs[4 * job] + (int64_t)a.jobs[4 * job + 1] * a.ny;
    }
    // ---- stages 1-3: the group loads the window's pixels (coalesced down
    //      the columns), reduces the window means in FP64, and stores
    //      apod * (x - mean) into the plane; masked pixels enter as zero and
    //      leave the mean (load_windows!, src/correlators.jl:188-263). The
    //      mean is the exact sum over n rounded once, where the reference
    //      folds in Float32 left to right; the two differ by a few ulp.
    bool bad;
    if (ROWSCAN && N2 > 1)
      for (int r = gt; r < N; r += G) rmax[r] = 0u;  // raised by the last inverse pass, barriers later
    if constexpr (SRCH) {
      // enlarged search area (load_windows!, src/correlators.jl:229-262):
      // the W x W frame-B area starts (W - win) / 2 before the window on
      // both axes; frame A enters only inside the centred window, apodized
      // and less its own mean, frame B everywhere, less its mean, without
      // apodization; a masked pixel is zero in both and leaves both means
      const int wa = a.win, oa = (W - wa) / 2;
      const int64_t r0 = rs - oa, c0 = cs - oa;
      // VIA: pixels in batches of LB, stored raw until the means are known
      constexpr int LB = C::VIA ? 8 : EPT;
      float2 z[LB];
      bool mk[EPT];  // masked, or past the area
      double sa = 0.0, sb = 0.0, na = 0.0, nb = 0.0;
#pragma unroll
      for (int i0 = 0; i0 < EPT; i0 += LB) {
#pragma unroll
        for (int i = 0; i < LB; ++i) {
          const int e = gt + (i0 + i) * G, p = e % W, q = e / W;
          const bool in = W * W % (G * LB) == 0 || e < W * W;
          const bool ina = (unsigned)(p - oa) < (unsigned)wa && (unsigned)(q - oa) < (unsigned)wa;
          const int64_t off = (r0 + p) + (c0 + q) * ld;
          z[i] = make_float2(ld_stream_if(A + off, in && ina), ld_stream_if(B + off, in));
          const bool m = !in || ld_stream_if(M + off, in && M) != 0;
          if (i0 + i < EPT) mk[i0 + i] = m;
        }
#pragma unroll
        for (int i = 0; i < LB && i0 + i < EPT; ++i) {
          const int e = gt + (i0 + i) * G, p = e % W, q = e / W;
          const bool ina = (unsigned)(p - oa) < (unsigned)wa && (unsigned)(q - oa) < (unsigned)wa;
          const bool m = mk[i0 + i];
          sb += (double)(m ? 0.f : z[i].y);
          sa += (double)(m ? 0.f : z[i].x);  // 0 outside the window
          nb += m ? 0.0 : 1.0;
          na += m || !ina ? 0.0 : 1.0;
          if (C::VIA && (W * W % (G * LB) == 0 || e < W * W)) P[q * LD + p] = z[i];
        }
      }
      const unsigned gm = grp_mask(G);
#pragma unroll
      for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1) {
        sa += __shfl_xor_sync(gm, sa, o);
        sb += __shfl_xor_sync(gm, sb, o);
        na += __shfl_xor_sync(gm, na, o);
        nb += __shfl_xor_sync(gm, nb, o);
      }
      double ta = sa, tb = sb, tna = na, tnb = nb;
      if (G > 32) {
        if (lane == 0) {
          part[4 * gw] = sa;
          part[4 * gw + 1] = sb;
          part[4 * gw + 2] = na;
          part[4 * gw + 3] = nb;
        }
        grp_sync(bar, G);
        ta = tb = tna = tnb = 0.0;
        for (int k = 0; k < G / 32; ++k) {
          ta += part[4 * k];
          tb += part[4 * k + 1];
          tna += part[4 * k + 2];
          tnb += part[4 * k + 3];
        }
      }
      const float ma = tna > 0 ? (float)(ta / tna) : 0.f, mb = tnb > 0 ? (float)(tb / tnb) : 0.f;
      bad = !(isfinite(ta) && isfinite(tb));
#pragma unroll
      for (int i = 0; i < EPT; ++i) {
        const int e = gt + i * G;
        if (e < W * W) {
          const int p = e % W, q = e / W;
          const bool ina = (unsigned)(p - oa) < (unsigned)wa && (unsigned)(q - oa) < (unsigned)wa;
          const float2 x = C::VIA ? P[q * LD + p] : z[i % LB];
          float2 v = make_float2(0.f, 0.f);
          if (!(mk[i] || bad)) {
            v.y = x.y - mb;
            if (ina) v.x = ld_keep(a.apod + (p - oa) + (q - oa) * wa) * (x.x - ma);
          }
          P[q * LD + p] = v;
        }
      }
    } else {
      // in batches of LB pixel pairs, a batch's loads in flight together
      constexpr int LB = C::VIA ? 8 : EPT;
      float2 z[LB];
      uint32_t mk[(EPT + 31) / 32] = {};  // masked, or past the window
      double sa = 0.0, sb = 0.0, cnt = 0.0;
      auto load = [&](int i0) {
        const int64_t w0 = (int64_t)rs + (int64_t)cs * ld;
        uint32_t m = 0u;
#pragma unroll
        for (int i = 0; i < LB; ++i) {
          const int e = gt + (i0 + i) * G;
          const bool in = W * W % (G * LB) == 0 || e < W * W;
          const int64_t off = w0 + e % W + (int64_t)(e / W) * ld;
          z[i] = make_float2(ld_stream_if(A + off, in), ld_stream_if(B + off, in));
          m |= (uint32_t)(!in || ld_stream_if(M + off, in && M) != 0) << i;
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
          const bool k = m >> i & 1u;
          sa += (double)(k ? 0.f : z[i].x);
          sb += (double)(k ? 0.f : z[i].y);
          cnt += k ? 0.0 : 1.0;
        }
        return m;
      };
      if constexpr (C::VIA) {
#pragma unroll
        for (int i0 = 0; i0 < EPT; i0 += LB) {
          mk[i0 / 32] |= load(i0) << (i0 % 32);
#pragma unroll
          for (int i = 0; i < LB; ++i) {
            const int e = gt + (i0 + i) * G;
            if (W * W % (G * LB) == 0 || e < W * W) P[e / W * LD + e % W] = z[i];
          }
        }
      } else {
        mk[0] = load(0);
      }
      const unsigned gm = grp_mask(G);
#pragma unroll
      for (int o = (G < 32 ? G : 32) / 2; o > 0; o >>= 1) {
        sa += __shfl_xor_sync(gm, sa, o);
        sb += __shfl_xor_sync(gm, sb, o);
        cnt += __shfl_xor_sync(gm, cnt, o);
      }
      double ta = sa, tb = sb, tn = cnt;
      if (G > 32) {
        if (lane == 0) {
          part[3 * gw] = sa;
          part[3 * gw + 1] = sb;
          part[3 * gw + 2] = cnt;
        }
        grp_sync(bar, G);
        ta = tb = tn = 0.0;
        for (int k = 0; k < G / 32; ++k) {
          ta += part[3 * k];
          tb += part[3 * k + 1];
          tn += part[3 * k + 2];
        }
      }
      const float ma = tn > 0 ? (float)(ta / tn) : 0.f, mb = tn > 0 ? (float)(tb / tn) : 0.f;
      bad = !(isfinite(ta) && isfinite(tb));  // the window holds NaN or Inf
#pragma unroll
      for (int i = 0; i < EPT; ++i) {
        const int e = gt + i * G;
        if (W * W % G == 0 || e < W * W) {
          float2* c = P + e / W * LD + e % W;
          const float ap = ld_keep(a.apod + e);
          const float2 v = C::VIA ? *c : z[i % LB];
          *c = (mk[i / 32] >> (i % 32) & 1u) || bad ? make_float2(0.f, 0.f) : make_float2(ap * (v.x - ma), ap * (v.y - mb));
        }
      }
    }
    grp_sync(bar, G);

    // ---- stage 4: forward transform along p (only the W data columns)
    for (int it = gt; it < W * N2; it += G) {
      const int q = it % W, n2 = it / W;
      float2* L = P + q * LD;
      float2 x[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) x[n1] = n1 < C::NZ1 ? L[N2 * n1 + n2] : make_float2(0.f, 0.f);
      RDFT<N1, false>::run(x, C::NZ1);
      if (N2 > 1) {
#pragma unroll
        for (int k1 = 1; k1 < N1; ++k1) x[k1] = cmul(x[k1], tw[n2 * k1]);
      }
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) L[N2 * k1 + n2] = x[k1];
    }
    if (N2 > 1) {
      grp_sync(bar, G);
      for (int it = gt; it < W * N1; it += G) {
        const int q = it % W, k1 = it / W;
        float2* L = P + q * LD + N2 * k1;
        float2 x[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) x[n2] = L[n2];
        RDFT<N2, false>::run(x, N2);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) L[k2] = x[k2];
      }
    }
    grp_sync(bar, G);
    // ---- stage 5: forward transform along q for every row p
    for (int it = gt; it < N * N2; it += G) {
      const int p = it % N, n2 = it / N;
      float2* L = P + p;
      float2 x[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) x[n1] = n1 < C::NZ1 ? L[(N2 * n1 + n2) * LD] : make_float2(0.f, 0.f);
      RDFT<N1, false>::run(x, C::NZ1);
      if (N2 > 1) {
#pragma unroll
        for (int k1 = 1; k1 < N1; ++k1) x[k1] = cmul(x[k1], tw[n2 * k1]);
      }
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) L[(N2 * k1 + n2) * LD] = x[k1];
    }
    grp_sync(bar, G);
    // ---- stages 6-7: cross-power (or filtered phase) spectrum over Hermitian
    //      pairs (k, -k) and the inverse along p, on the canonical columns
    //      kq = 0..N/2 only (frequencies in storage order for N2 > 1, natural
    //      order otherwise); column -kq is conj of column kq and is not stored.
    //      For N <= 32 every canonical column's spectrum is formed in place
    //      here: folding it into the single-pass inverse costs more registers
    //      than the separate pass costs time.
    if constexpr (N2 == 1 && G <= N && N % G == 0) {
      // each thread owns rows ap = gt + j G (j < N / G) of every canonical
      // column; the columns are unrolled, so every address is the row's base
      // plus a constant, and CB columns' operands are loaded before any of
      // their results is stored (no item reads a cell another item writes:
      // column -c is read only, and a self-paired column's rows ap and -ap
      // belong to one item)
      constexpr int RPT = G <= N ? N / G : 1, CB = RPT >= 2 ? 2 : 4;
      int ra[RPT], rb[RPT];
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        ra[j] = gt + j * G;
        rb[j] = (N - ra[j]) % N;
      }
#pragma unroll
      for (int c0 = 0; c0 < NC; c0 += CB) {
        float2 xa[CB][RPT], xb[CB][RPT];
        float wk[CB][RPT];
#pragma unroll
        for (int u = 0; u < CB; ++u) {
          const int c = c0 + u, cb = (N - c) % N;
          if (c < NC) {
#pragma unroll
            for (int j = 0; j < RPT; ++j) {
              if (c == cb && ra[j] > rb[j]) continue;  // a self pair is done by its upper row
              xa[u][j] = P[c * LD + ra[j]];
              xb[u][j] = P[cb * LD + rb[j]];
              wk[u][j] = method == 1 ? ld_keep(a.phasew + c * N + ra[j]) : 1.f;
            }
          }
        }
#pragma unroll
        for (int u = 0; u < CB; ++u) {
          const int c = c0 + u, cb = (N - c) % N;
          if (c < NC) {
#pragma unroll
            for (int j = 0; j < RPT; ++j) {
              if (c == cb && ra[j] > rb[j]) continue;
              const float2 S = cross_spectrum(xa[u][j], xb[u][j], method, wk[u][j]);
              P[c * LD + ra[j]] = S;
              if (c == cb) P[c * LD + rb[j]] = make_float2(S.x, -S.y);
            }
          }
        }
      }
    } else if constexpr (N2 == 1) {
      // items (row ap, canonical column c) in batches of SB per thread: the
      // batch's operands are loaded before any of its results is stored (no
      // item reads a cell another item writes: column -c is read only, and a
      // self-paired column's rows ap and -ap belong to one item)
      constexpr int SB = 4, NIT = NC * N;  // (batches of 8 were slower: registers)
#pragma unroll 1
      for (int it0 = gt; it0 < NIT; it0 += SB * G) {
        float2 xa[SB], xb[SB];
        int ia[SB], ib[SB];
        bool on[SB], self[SB];
        float wk[SB];
#pragma unroll
        for (int u = 0; u < SB; ++u) {
          const int it = it0 + u * G;
          const int ap = it % N, c = it / N, bq = (N - c) % N, bp = (N - ap) % N;
          self[u] = c == bq;
          on[u] = it < NIT && !(self[u] && ap > bp);  // a self pair is done by its upper row
          ia[u] = c * LD + ap;
          ib[u] = bq * LD + bp;
          wk[u] = on[u] && method == 1 ? ld_keep(a.phasew + c * N + ap) : 1.f;
          if (on[u]) {
            xa[u] = P[ia[u]];
            xb[u] = P[ib[u]];
          }
        }
#pragma unroll
        for (int u = 0; u < SB; ++u)
          if (on[u]) {
            const float2 S = cross_spectrum(xa[u], xb[u], method, wk[u]);
            P[ia[u]] = S;
            if (self[u]) P[ib[u]] = make_float2(S.x, -S.y);
          }
      }
    } else {
      // For N2 > 1 the second pass along q forms the spectrum from its own
      // registers. Slot k2 of group k1 holds frequency k1 + N1 k2, canonical
      // for k2 < N2/2 (and N2/2 of group 0); its negation is slot N2-1-k2 of
      // group N1-k1 (slot N2-k2 of group 0 for group 0) in row -kp. So an item
      // takes group ga of row ra and group gb = -ga of row rb = -ra, reads
      // what it overwrites and nothing that another item writes: all rows for
      // ga = 1 .. N1/2-1, and for ga = 0 and N1/2 (their own negations) a row
      // of each pair, the self-negated rows 0 and N/2 together. Rows -ra of
      // consecutive ra are consecutive too. A separate spectrum step read and
      // wrote the whole plane once more, 4 to 5 % of a padded window's time: 12.8
      // ns at 48 points against 12.3; 64: 22.3 and 21.3; 96: 53.2 and 51.0; 128:
      // 102 and 97 (11.7, 19.1, 49 and 93 with the later steps).
      constexpr int h2 = N2 / 2, HN = N1 / 2;
#pragma unroll 1
      for (int it = gt; it < N * HN; it += G) {
        int ga, gb, ra, rb;
        bool self = false;
        if (it < N * (HN - 1)) {
          ga = 1 + it / N;
          gb = N1 - ga;
          ra = it % N;
          rb = ra < N2 ? (N2 - ra) % N2 : N + N2 - 1 - ra;
        } else {
          const int e = it - N * (HN - 1), r = e % H;
          ga = gb = e < H ? 0 : HN;
          self = r == 0;  // rows 0 (kp = 0) and h2 (kp = N/2)
          ra = r < h2 ? r : N2 + r - h2;
          rb = self ? h2 : (ra < N2 ? N2 - ra : N + N2 - 1 - ra);
        }
        float2* La = P + ra + N2 * ga * LD;
        float2* Lb = P + rb + N2 * gb * LD;
        float2 xa[N2], xb[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) {
          xa[n2] = La[n2 * LD];
          xb[n2] = Lb[n2 * LD];
        }
        RDFT<N2, false>::run(xa, N2);
        RDFT<N2, false>::run(xb, N2);
        // the filter weight of canonical column c = g + N1 k2 at row r
        auto weight = [&](int g, int k2, int r) {
          return method == 1 ? ld_keep(a.phasew + (g + N1 * k2) * N + r / N2 + N1 * (r % N2)) : 1.f;
        };
        if (ga != 0) {
          auto pair = [&](const float2(&ya)[N2], const float2(&yb)[N2]) {
#pragma unroll
            for (int k2 = 0; k2 < h2; ++k2) {
              La[k2 * LD] = cross_spectrum(xa[k2], ya[N2 - 1 - k2], method, weight(ga, k2, ra));
              Lb[k2 * LD] = cross_spectrum(xb[k2], yb[N2 - 1 - k2], method, weight(gb, k2, rb));
            }
          };
          if (self) pair(xa, xb);
          else pair(xb, xa);
        } else {
          auto pair = [&](const float2(&ya)[N2], const float2(&yb)[N2]) {
#pragma unroll
            for (int k2 = 0; k2 <= h2; ++k2) {
              const float2 S = cross_spectrum(xa[k2], ya[(N2 - k2) % N2], method, weight(0, k2, ra));
              if (k2 != 0 && k2 != h2) {
                La[k2 * LD] = S;
                Lb[k2 * LD] = cross_spectrum(xb[k2], yb[(N2 - k2) % N2], method, weight(0, k2, rb));
              } else if (!self) {  // columns 0 and N/2 are their own negations
                La[k2 * LD] = S;
                Lb[k2 * LD] = make_float2(S.x, -S.y);
              } else {
                const float2 T = cross_spectrum(xb[k2], yb[(N2 - k2) % N2], method, weight(0, k2, rb));
                La[k2 * LD] = make_float2(S.x, -S.y);
                Lb[k2 * LD] = make_float2(T.x, -T.y);
              }
            }
          };
          if (self) pair(xa, xb);
          else pair(xb, xa);
        }
      }
    }
    grp_sync(bar, G);
    if (N2 > 1) {
#pragma unroll 1
      for (int it = gt; it < NC * N1; it += G) {
        int c, k1;
        if (it >= H * N1) {  // column N/2 last
          c = H;
          k1 = it - H * N1;
        } else if (C::ROT) {
          constexpr int U = N2 / 2 > 0 ? N2 / 2 : 1;
          const int w = it / U;
          c = N1 * (it % U) + w % N1;
          k1 = w / N1;
        } else if (N2 == 6) {  // columns of u = 0, 1, then those of u = 2
          const bool lo = it < 2 * N1 * N1;
          const int e = lo ? it : it - 2 * N1 * N1;
          c = lo ? e % (2 * N1) : 2 * N1 + e % N1;
          k1 = lo ? e / (2 * N1) : e / N1;
        } else {
          c = it % H;
          k1 = it / H;
        }
        float2* L = P + s_canon[c] * LD + N2 * k1;
        const int swap = C::rot(c % N1);  // N2/2: the halves of the group change places
        float2* L0 = L + swap;            // slots of k2 < N2/2
        float2* L1 = L - swap;
        const uint32_t sign = swap ? 0x80000000u : 0u;
        float2 x[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) x[k2] = (k2 < N2 / 2 ? L0 : L1)[k2];
        RDFT<N2, true>::run(x, N2);
#pragma unroll
        for (int n2 = 1; n2 < N2; ++n2) {
          const float2 t = tw[n2 * k1];
          if (C::ROT && n2 % 2 == 1)  // the sign bits: a negated operand would change how the product is contracted
            x[n2] = make_float2(__uint_as_float(__float_as_uint(x[n2].x) ^ sign),
                                __uint_as_float(__float_as_uint(x[n2].y) ^ sign));
          x[n2] = cmul(x[n2], make_float2(t.x, -t.y));
        }
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) (n2 < N2 / 2 ? L0 : L1)[n2] = x[n2];
      }
      grp_sync(bar, G);
    }
#pragma unroll 1
    //      With N2 = 1 the two self-paired columns kq = 0 and N/2, whose
    //      results are real, share one transform as col0 + i col(N/2) (real
    //      part: column 0, imaginary part: column N/2): H items in all.
    //      With N2 > 1 consecutive threads take consecutive n2 of one column
    //      (the canonical columns sit N2 storage columns apart, which alias
    //      to two banks; rows n2 of one column do not).
    for (int it = gt; it < (N2 == 1 ? H : NC * N2); it += G) {
      const bool pk = N2 == 1 && it == 0;
      const int c = N2 == 1 ? it : it / N2, n2 = N2 == 1 ? 0 : it % N2;
      const int aq = N2 == 1 ? c : s_canon[c];
      float2* L = P + aq * LD;
      float2* Lb = P + H * LD;  // column N/2, for the packed item only
      float2 x[N1];
#pragma unroll
      for (int k1 = 0; k1 < N1; ++k1) {
        const float2 u = L[N2 * k1 + n2];
        if (pk) {
          const float2 v = Lb[k1];
          x[k1] = make_float2(u.x - v.y, u.y + v.x);
        } else {
          x[k1] = u;
        }
      }
      RDFT<N1, true>::run(x, N1);
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) {
        if (!C::keep(n1)) continue;
        if (pk) {
          L[n1] = make_float2(x[n1].x, 0.f);
          Lb[n1] = make_float2(x[n1].y, 0.f);
        } else {
          L[N2 * n1 + n2] = x[n1];
        }
      }
    }
    grp_sync(bar, G);
    // ---- stage 8: inverse along q for the rows R needs: fftshifted rows
    //      blo..bhi (the overlap gain is zero on every other row, so R is
    //      exactly 0 there), taken in pairs (blo + t, blo + t + nh) packed as
    //      T(p) + i T(p'). Column -kq of T is the conjugate of column kq, so
    //      only the canonical columns were stored; each value read (u, v of
    //      the two rows) gives u + i v for kq and conj(u) + i conj(v) for
    //      -kq. The normalised, gain-weighted magnitudes are held in registers
    //      across a barrier, then written as the real plane R over the
    //      complex one.
    if constexpr (N2 > 1) {
      // The first pass takes the groups k1 = j and N1 - j (0 and N1/2 for
      // j = 0) of a row pair together: slot k2 of group k1 (frequency
      // k1 + N1 k2) is canonical for k2 < N2/2 (and N2/2 of group 0), and the
      // other half of each group mirrors the first half of the other (of
      // itself for j = 0), so the item reads what it overwrites and nothing
      // that another item writes.
      constexpr int h2 = N2 / 2, HN = N1 / 2;
#pragma unroll 1
      for (int it = gt; it < nh * HN; it += G) {
        const int j = (it * inv_nh) >> 16, t = it - j * nh;
        const bool hasb = t + nh < nb, j0 = j == 0;
        const int pa = (blo + t + H) % N, pb = hasb ? (blo + t + nh + H) % N : pa;
        const int ga = N2 * j, gb = N2 * (j0 ? HN : N1 - j);
        // the rows' slots in the columns of groups j and N1 - j
        const int kb = j0 ? HN : N1 - j, ta = C::rot(j), tb = C::rot(kb);
        float2 x1[N2], x2[N2], ma[h2 + 1], mb[h2];
        auto row_pair = [&](int slot, int t, float2& direct, float2& mirror) {
          const float2 u = P[(pa ^ t) + slot * LD];
          const float2 v = hasb ? P[(pb ^ t) + slot * LD] : make_float2(0.f, 0.f);
          direct = make_float2(u.x - v.y, u.y + v.x);
          mirror = make_float2(u.x + v.y, v.x - u.y);
        };
#pragma unroll
        for (int k2 = 0; k2 < h2; ++k2) {
          row_pair(ga + k2, ta, x1[k2], ma[k2]);
          row_pair(gb + k2, tb, x2[k2], mb[k2]);
        }
        float2 mid = make_float2(0.f, 0.f);
        if (j0) row_pair(h2, 0, mid, ma[h2]);
#pragma unroll
        for (int k2 = h2; k2 < N2; ++k2) {
          const float2 own = k2 == h2 ? mid : ma[N2 - k2];
          x1[k2] = j0 ? own : mb[N2 - 1 - k2];
          x2[k2] = j0 ? mb[N2 - 1 - k2] : ma[N2 - 1 - k2];
        }
        RDFT<N2, true>::run(x1, N2);
        RDFT<N2, true>::run(x2, N2);
#pragma unroll
        for (int n2 = 1; n2 < N2; ++n2) {
          const float2 wa = tw[n2 * j], wb = tw[n2 * kb];
          x1[n2] = cmul(x1[n2], make_float2(wa.x, -wa.y));
          x2[n2] = cmul(x2[n2], make_float2(wb.x, -wb.y));
        }
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) {
          P[(pa ^ ta) + (ga + n2) * LD] = x1[n2];
          P[(pa ^ tb) + (gb + n2) * LD] = x2[n2];
        }
      }
      grp_sync(bar, G);
    }
    {
      float rv[IPT][2][N1];
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        const int it = gt + i * G;  // items (t, n2) at it = t + nh n2
        if (it < nh * N2) {
          const int n2 = N2 == 1 ? 0 : (it * inv_nh) >> 16, t = it - n2 * nh;
          const bool hasb = t + nh < nb;
          const int pa = (blo + t + H) % N, pb = hasb ? (blo + t + nh + H) % N : pa;
          const float2* La = P + pa;
          const float2* Lb = P + pb;
          float2 x[N1];
          if (N2 == 1) {
#pragma unroll
            for (int k1 = 0; k1 <= H; ++k1) {
              const float2 u = La[k1 * LD];
              const float2 v = hasb ? Lb[k1 * LD] : make_float2(0.f, 0.f);
              x[k1 % N1] = make_float2(u.x - v.y, u.y + v.x);
              if (k1 > 0 && k1 < H) x[(N - k1) % N1] = make_float2(u.x + v.y, v.x - u.y);
            }
          } else {
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) x[k1] = P[(pa ^ C::rot(k1)) + (N2 * k1 + n2) * LD];
          }
          RDFT<N1, true>::run(x, N1);
          const int ps0 = blo + t, ps1 = blo + t + nh;  // fftshifted rows of pa and pb
          float m0 = 0.f, m1 = 0.f;  // maxima of the two rows over this item's columns (a NaN drops out)
          const float* g0 = s_gain + (ps0 - (H - C::Q));  // row lag + Q of the gain table
          const float* g1 = s_gain + (hasb ? ps1 - (H - C::Q) : 0);
#pragma unroll
          for (int n1 = 0; n1 < N1; ++n1) {
            if (!C::keep(n1)) continue;
            const int q = N2 * n1 + n2, qs = (q + H) % N;
            float r0 = fabsf(x[n1].x) * scale, r1 = fabsf(x[n1].y) * scale;
            if (C::BOXED) {
              // columns past Q, which no lag is kept of, appear for N2 > 1 only
              const int gc = 2 * n1 < N1 ? q + C::Q : q + C::Q - N;
              if (N2 == 1 || (gc >= 0 && gc < GB)) {
                r0 *= g0[gc * GB];
                r1 *= g1[gc * GB];
              }
            }
            if (SRCH && (qs < blo || qs > bhi)) r0 = r1 = 0.f;  // lags outside the search range
            rv[i][0][n1] = r0;
            rv[i][1][n1] = r1;
            m0 = fmaxf(m0, r0);
            m1 = fmaxf(m1, r1);
          }
          if (!ROWSCAN) {
          } else if (N2 == 1) {
            rmax[ps0] = __float_as_uint(m0);
            if (hasb) rmax[ps1] = __float_as_uint(m1);
          } else {
            atomicMax(rmax + ps0, __float_as_uint(m0));
            if (hasb) atomicMax(rmax + ps1, __float_as_uint(m1));
          }
        }
      }
      grp_sync(bar, G);
#pragma unroll
      for (int i = 0; i < IPT; ++i) {
        const int it = gt + i * G;
        if (it < nh * N2) {
          const int n2 = N2 == 1 ? 0 : (it * inv_nh) >> 16, t = it - n2 * nh;
          const bool hasb = t + nh < nb;
          const int ps0 = blo + t, ps1 = blo + t + nh;
#pragma unroll
          for (int n1 = 0; n1 < N1; ++n1) {
            if (!C::keep(n1)) continue;
            const int qs = (N2 * n1 + n2 + H) % N;
            Rw[qs * LDR + ps0] = rv[i][0][n1];
            if (hasb) Rw[qs * LDR + ps1] = rv[i][1][n1];
          }
        }
      }
      if (!C::BOXED) {
        const int nz = N - nb;  // rows outside [blo, bhi]
        for (int j = gt; j < nz; j += G) {
          const int ps = j < blo ? j : j + nb;
#pragma unroll 4
          for (int qs = 0; qs < N; ++qs) Rw[qs * LDR + ps] = 0.f;
        }
      }
    }
    grp_sync(bar, G);
    if (a.planes) {
      float* dst = a.planes + job * (int64_t)(N * N);
      for (int it = gt; it < N * N; it += G) {
        const int p = it % N, q = it / N;
        const bool in = !C::BOXED || (p >= blo && p <= bhi && q >= blo && q <= bhi);
        const float r = in ? Rw[q * LDR + p] : 0.f;
        // ensemble: per-pair planes summed in pair order; a window with
        // non-finite data poisons its sum as the reference's NaN plane does
        const float rr = bad ? __int_as_float(0x7fc00000) : r;
        dst[q * N + p] = a.accumulate ? dst[q * N + p] + rr : rr;
      }
      if (a.accumulate) {  // ensemble planes are analysed once, after the last pair
        grp_sync(bar, G);
        continue;
      }
    }
    // ---- stage 9: peak analysis by the group (the output pointers are
    //      needed only when the outputs are formed here, not from a record)
    const bool defer = a.rec && a.finder == 0;
    uint32_t* gred = red + w * (G / 32) * 2 * KMAX;
    if (C::INLINE_ANALYSIS && K <= 4)
      analyze_body<4, FN, C::BOXED>(Rw, N, N, LDR, K, a.npeaks, a.finder, a.subpixel, gt, G, gred, true, s_vals + w * KMAX,
                            s_locs + w * 2 * KMAX, gid, job, defer ? nullptr : &pw, bad, bar, sp, a.rec, a.njobs, rmax,
                          list);
    else if (C::INLINE_ANALYSIS)
      analyze_body<KMAX, FN, C::BOXED>(Rw, N, N, LDR, K, a.npeaks, a.finder, a.subpixel, gt, G, gred, true, s_vals + w * KMAX,
                               s_locs + w * 2 * KMAX, gid, job, defer ? nullptr : &pw, bad, bar, sp, a.rec, a.njobs,
                               rmax, list);
    else
      analyze_group<FN, C::BOXED>(Rw, N, N, LDR, K, a.npeaks, a.finder, a.subpixel, gt, G, gred, true, s_vals + w * KMAX,
                          s_locs + w * 2 * KMAX, gid, job, defer ? nullptr : &pw, bad, bar, sp, a.rec, a.njobs, rmax,
                          list);
    grp_sync(bar, G);  // the plane is reused by the group's next window
  }
}

// ---------------------------------------------------------------------------
template <int N, int W, bool SRCH, int VAR, bool ANY = true>
static cudaError_t launch_nw(const CorrArgs& a, cudaStream_t s, int num_sms) {
  using C = CorrCfg<N, W, SRCH, VAR>;
  const size_t sm = C::smem();
  if (C::BOXED && !(a.gain && a.box_hi > 0 && a.box_lo >= N / 2 - C::Q && a.box_hi <= N / 2 + C::Q))
    return cudaErrorInvalidValue;
  static DeviceOnce attr;
  cudaError_t e = raise_smem_carveout(attr, correlate_kernel<N, W, SRCH, VAR, ANY>, sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, correlate_kernel<N, W, SRCH, VAR, ANY>, C::NT, sm);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int64_t units = (a.njobs + C::WPC - 1) / C::WPC;
  int64_t grid = (int64_t)per_sm * num_sms;
  if (grid > units) grid = units;
  if (grid < 1) grid = 1;
  correlate_kernel<N, W, SRCH, VAR, ANY><<<(unsigned)grid, C::NT, sm, s>>>(a);
  e = cudaGetLastError();
  if (e == cudaSuccess && a.rec && a.finder == 0 && !a.accumulate) e = launch_peak_epilogue(a, N, s, num_sms);
  return e;
}

// The variant of (N, W) that `a` asks for.
template <int N, int W> static cudaError_t launch_corr_nw(const CorrArgs& a, cudaStream_t s, int num_sms) {
  if (a.win > 0 && a.win < W) return launch_nw<N, W, true, 0>(a, s, num_sms);
  // 16 and 32 points: several windows per warp (hh_corr_seg.cuh) for the
  // regional-maximum finder and the ensemble sums; the exclusion finder, which
  // ranks its peaks in place, keeps this file's kernel. ns per window on one
  // 2048^2 pair, this kernel / that one: 8 px padded 2.8 / 0.96, 16 px padded
  // 4.5 / 3.3, 16 px 3.8 / 2.0, 32 px 8.6 / 6.6. While an SM holds all its
  // windows at once, a warp each, this kernel is the faster one where the peaks
  // are searched in the whole plane: us, this / that, 16 px 100 windows 24 / 34,
  // 3000 33 / 34, 5000 42 / 36; 32 px, up to 4 peaks, 100 windows 25 / 28, 2368
  // 35 / 36, 3000 42 / 38; with more peaks, whose lists take the registers, 100
  // windows 41 / 62, 6000 79 / 82, 20000 226 / 214. Padded windows, whose box is
  // small, stay within 2 us of each other there, and planes that are only summed
  // too, but for 16 px (289 windows, 8 pairs 103 / 117 us, 1296 windows 128 / 120).
  if constexpr (N == 16 || N == 32) {
    const int from = W < N ? 0 : a.accumulate ? (N == 16 ? 6 : 0) : N == 16 ? 24 : a.npeaks <= 4 ? 16 : 64;  // windows per SM
    if (a.variant == 0 && seg_serves(a) && a.njobs > (int64_t)from * num_sms) return launch_seg<N, W>(a, s, num_sms);
  }
  switch (a.variant) {
    case 1: return launch_nw<N, W, false, 1>(a, s, num_sms);
    case 2: return launch_nw<N, W, false, 2>(a, s, num_sms);
    case 3: return launch_nw<N, W, false, 3>(a, s, num_sms);
    case 4: return launch_nw<N, W, false, 4>(a, s, num_sms);
    default:
      return a.method == 1 ? launch_nw<N, W, false, 0>(a, s, num_sms) : launch_nw<N, W, false, 0, false>(a, s, num_sms);
  }
}

// The launch of one FFT size: each size is a translation unit of its own
// (k_corr_<N>.cu), because the five variants of all sizes together take
// minutes to compile.
#define HH_CORR_SIZE(N)                                                                                       \
  cudaError_t launch_corr_##N(const CorrArgs& a, int W, cudaStream_t s, int num_sms) {                       \
    return W == N ? launch_corr_nw<N, N>(a, s, num_sms) : launch_corr_nw<N, N / 2>(a, s, num_sms);            \
  }

}  // namespace hh
