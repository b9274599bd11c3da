// Fused window correlation for 16- and 32-point FFTs: several windows per
// warp, in lockstep.
//
// Every stage of an N-point plane whose lines fit a lane's registers has N/2
// items or a multiple of it (N/2 packed canonical columns of the inverse, at
// most N/2 row pairs, N rows and W columns forward), so a window takes
// SEG = N/2 lanes and a warp carries 2 (32 points) or 4 (16 points) windows
// with no lane idle, where a warp or half-warp per window left half of them
// idle in the inverse. The windows of a warp advance together: all
// collectives are full-warp shuffles and ballots, so no half waits for the
// other's loop. What else differs from the general fused kernel:
//   - the raw pixels go straight to the plane and the column transform applies
//     mean and apodization as it reads them (no pixel is held in registers);
//   - a lane transforms row p while the lane of row -p transforms that one
//     (rows are dealt in sets closed under negation), so the spectrum
//     S(p, q) = conj(FA) FB needs Z(-p, -q) from one shuffle, not from a
//     plane that holds both rows, and only the canonical columns are stored;
//   - the two real-valued columns 0 and N/2 of the inverse live packed in
//     column 0 from the spectrum to the last pass, so a plane has N/2 columns
//     (W when that is more): half the shared memory, 4 CTAs of 4 warps per SM
//     instead of 3.
// The arithmetic of every value is the general kernel's, so the planes are
// the same bit for bit. The pixel loads of a batch carry no branch (the image
// mask's bytes are gathered apart): with one per pixel the loads went out one
// by one, and a third of a warp's time was the wait for them (32-point padded
// windows 4.6 -> 3.5 ns, unpadded 12.1 -> 7.3; 3.3 and 6.6 with packed complex
// sums, cadd2). Bound by issue and latency (half the issue slots used at 16 to
// 20 warps per SM); which launches take it, and their times, in launch_corr_nw.
#pragma once
#include "hh_attr.h"
#include "hh_corr_peaks.cuh"

namespace hh {

template <int N, int W> struct SegCfg {
  static constexpr int H = N / 2, Q = N / 4, SEG = H, HS = SEG / 2;
  static constexpr int WPW = 32 / SEG;         // windows per warp
  static constexpr int NT = 128, WIN = NT / SEG;  // windows per CTA
  static constexpr bool BOXED = 2 * W == N;    // padded: only lags |lag| <= Q are kept (CorrCfg::BOXED)
  static constexpr bool keep(int n) { return !BOXED || n <= Q || n >= N - Q; }
  static constexpr int CR = W / SEG, RR = N / SEG;  // column and row rounds
  static constexpr int LD = N + 1;             // of the complex plane (float2) and the real one (float)
  static constexpr int COLS = W > H ? W : H;
  // the windows of a half-warp (64-bit accesses) and of a warp (32-bit ones) start 16 banks apart
  static constexpr int PS = (COLS * LD + 15) / 16 * 16 + 8;
  static constexpr int MINB = W == 32 ? 3 : (N == 16 ? 5 : 4);
  static constexpr size_t off_apod = (size_t)WIN * PS * sizeof(float2);
  static constexpr size_t off_gain = off_apod + (size_t)W * (W + 1) * sizeof(float);
  static constexpr size_t off_rmax = off_gain + (BOXED ? (2 * Q + 1) * (2 * Q + 1) * sizeof(float) : 0);
  static constexpr size_t off_list = off_rmax + (BOXED ? 0 : WIN * N * sizeof(uint32_t));
  static constexpr size_t off_vals = off_list + (BOXED ? 0 : WIN * 2 * SEG * sizeof(uint16_t));
  static constexpr size_t off_locs = off_vals + WIN * KMAX * sizeof(float);
  static constexpr size_t off_map = off_locs + WIN * 2 * KMAX * sizeof(int);
  static constexpr size_t smem() { return off_map + rec_words(KMAX) * sizeof(uint32_t); }
  static_assert(N * LD * sizeof(float) <= PS * sizeof(float2), "the real plane fits in the complex one");
  static_assert(W % SEG == 0 && N == 2 * SEG, "lines are dealt in whole rounds");
};

// maximum over the SEG lanes of a segment
template <int SEG> __device__ __forceinline__ uint32_t seg_max(uint32_t v) {
#pragma unroll
  for (int o = SEG / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// warp_topk for segments in lockstep: lane m < n of each segment receives the
// segment's m-th best key.
template <int SEG, class TK>
__device__ __forceinline__ int seg_topk(TK& tk, int K, int l, uint32_t& mh, uint32_t& ml) {
  constexpr unsigned FULL = 0xffffffffu, ALL = (1u << SEG) - 1u;
  const int sb = (threadIdx.x & 31) & ~(SEG - 1);
  int n = 0;
  mh = ml = 0u;
  for (int round = 0; round < K; ++round) {
    const uint32_t h = tk.hi[0], w = seg_max<SEG>(h);
    bool mine = w != 0u && h == w;
    unsigned b = (__ballot_sync(FULL, mine) >> sb) & ALL;
    if (__any_sync(FULL, __popc(b) > 1)) {  // equal values: the smaller index wins
      const uint32_t lo = mine ? tk.lo[0] : 0u, wl = seg_max<SEG>(lo);
      mine = mine && lo == wl;
      b = (__ballot_sync(FULL, mine) >> sb) & ALL;
    }
    const uint32_t wl = __shfl_sync(FULL, tk.lo[0], sb + (b ? __ffs(b) - 1 : 0));
    if (mine) tk.pop();
    if (l == round) {
      mh = w;
      ml = wl;
    }
    n += w != 0u;
  }
  return n;
}

// scan_rows for segments in lockstep (the whole plane is the box).
template <int N, class TK>
__device__ __forceinline__ void seg_scan_rows(TK& tk, const float* R, int K, const uint32_t* rmax, uint16_t* list,
                                              int l, bool scan) {
  constexpr int SEG = N / 2, LD = N + 1;
  constexpr unsigned FULL = 0xffffffffu, ALL = (1u << SEG) - 1u;
  const int sb = (threadIdx.x & 31) & ~(SEG - 1);
  uint32_t M[2], cand[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int r = l + j * SEG;
    M[j] = rmax[r];
    const uint32_t up = r > 0 ? rmax[r - 1] : 0u, dn = r < N - 1 ? rmax[r + 1] : 0u;
    cand[j] = M[j] > up && M[j] > dn ? M[j] : 0u;
  }
  uint32_t thr = 0u;
  bool more = true;  // a segment that runs out of candidates keeps bound 0
  for (int k = 0; k < K; ++k) {
    const uint32_t t = seg_max<SEG>(max(cand[0], cand[1]));
    more = more && t != 0u;
    thr = more ? t : 0u;
#pragma unroll
    for (int j = 0; j < 2; ++j) cand[j] = cand[j] == t ? 0u : cand[j];
  }
  auto test = [&](int e) {
    const int r = e % N, c = e / N;
    const float* p = R + c * LD + r;
    const float x = __int_as_float(0x7fc00000), v = *p;
    const bool hu = r > 0, hd = r < N - 1, hl = c > 0, hr = c < N - 1;
    const float ul = hu && hl ? p[-LD - 1] : x, lt = hl ? p[-LD] : x, dl = hd && hl ? p[-LD + 1] : x;
    const float u = hu ? p[-1] : x, d = hd ? p[1] : x;
    const float ur = hu && hr ? p[LD - 1] : x, rt = hr ? p[LD] : x, dr = hd && hr ? p[LD + 1] : x;
    const float b = fmaxf(fmaxf(ul, lt), fmaxf(dl, u)), t = fmaxf(fmaxf(ur, rt), fmaxf(dr, d));
    if (!isnan(v) && !(b > v) && !(t >= v)) tk.insert(fkey(v), ~(uint32_t)e, K);
  };
  uint32_t rows = ((__ballot_sync(FULL, scan && M[0] >= thr) >> sb) & ALL) |
                  (((__ballot_sync(FULL, scan && M[1] >= thr) >> sb) & ALL) << SEG);
  int cnt = 0;
  while (__any_sync(FULL, rows != 0u)) {
    const bool act = rows != 0u;
    const int r = act ? __ffs(rows) - 1 : 0;
    rows &= rows - 1;
    uint32_t v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) v[i] = __float_as_uint(R[(l + SEG * i) * LD + r]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const bool in = act && v[i] >= thr;
      const unsigned b = (__ballot_sync(FULL, in) >> sb) & ALL;
      if (in) list[cnt + __popc(b & ((1u << l) - 1u))] = (uint16_t)(r + (l + SEG * i) * N);
      cnt += __popc(b);
      if (__any_sync(FULL, cnt >= SEG)) {  // a full round of tests; the rest moves down
        __syncwarp();
        const bool f = cnt >= SEG;
        if (f) test(list[l]);
        const uint16_t q = list[SEG + l];
        __syncwarp();
        if (f) {
          list[l] = q;
          cnt -= SEG;
        }
        __syncwarp();  // past the entries left, the next rows write these words again, by other lanes
      }
    }
  }
  __syncwarp();
  if (l < cnt) test(list[l]);
}

template <int N, int W, int KC, bool PHASE>
__global__ void __launch_bounds__(SegCfg<N, W>::NT, SegCfg<N, W>::MINB) correlate_seg_kernel(const CorrArgs a) {
  using C = SegCfg<N, W>;
  constexpr int SEG = C::SEG, HS = C::HS, WPW = C::WPW, LD = C::LD, H = C::H, Q = C::Q;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* sap = reinterpret_cast<float*>(smem_raw + C::off_apod);  // column q at q (W + 1): lanes on columns
  float* s_gain = reinterpret_cast<float*>(smem_raw + C::off_gain);
  uint32_t* s_map = reinterpret_cast<uint32_t*>(smem_raw + C::off_map);
  const int tid = threadIdx.x, lane = tid & 31, l = lane & (SEG - 1), w = tid / SEG, sb = lane & ~(SEG - 1);
  float2* P = reinterpret_cast<float2*>(smem_raw) + w * C::PS;
  float* Rw = reinterpret_cast<float*>(P);
  uint32_t* rmax = reinterpret_cast<uint32_t*>(smem_raw + C::off_rmax) + w * N;
  uint16_t* list = reinterpret_cast<uint16_t*>(smem_raw + C::off_list) + w * 2 * SEG;
  float* s_vals = reinterpret_cast<float*>(smem_raw + C::off_vals) + w * KMAX;
  int* s_locs = reinterpret_cast<int*>(smem_raw + C::off_locs) + w * 2 * KMAX;
  const int K = a.npeaks > 2 ? a.npeaks : 2, nw = rec_words(K);

  for (int m = tid; m < W * W; m += C::NT) sap[m % W + m / W * (W + 1)] = a.apod[m];
  constexpr int GB = 2 * Q + 1;  // the gain of the kept lags
  if (C::BOXED)
    for (int m = tid; m < GB * GB; m += C::NT) s_gain[m] = a.gain[H - Q + m % GB + (H - Q + m / GB) * N];
  // what word wd of a peak record holds: its peak m, and for a patch cell the
  // offset from the peak (+ 2 per axis)
  for (int wd = tid; wd < nw; wd += C::NT) {
    uint32_t e = 0u;
    if (wd >= 1 + 3 * K) {
      const int x = wd - 1 - 3 * K, m = x < 25 ? 0 : 1 + (x - 25) / 9, cell = x < 25 ? x : (x - 25) % 9;
      const int h = m == 0 ? 2 : 1, s = 2 * h + 1;
      e = (uint32_t)m | (uint32_t)(cell % s - h + 2) << 8 | (uint32_t)(cell / s - h + 2) << 16;
    }
    s_map[wd] = e;
  }
  __syncthreads();  // the only CTA-wide barrier

  const float scale = 1.0f / (float)(N * N);
  const int blo = C::BOXED ? a.box_lo : 0, bhi = C::BOXED ? a.box_hi : N - 1;
  const int nb = bhi - blo + 1, nh = (nb + 1) / 2;
  const int64_t units = (a.njobs + WPW - 1) / WPW;
  for (int64_t unit = (int64_t)blockIdx.x * (C::NT / 32) + (tid >> 5); unit < units;
       unit += (int64_t)gridDim.x * (C::NT / 32)) {
    const int64_t job = unit * WPW + lane / SEG;
    bool on = job < a.njobs;
    int rs = 0, cs = 0;
    const float* A = a.A;
    const float* B = a.B;
    const uint8_t* M = a.mask;
    int64_t ld = a.ld;
    if (on) {
      rs = a.jobs[4 * job + 2];
      cs = a.jobs[4 * job + 3];
      if (a.bp) {
        const int p = a.jobs[4 * job];
        const BPair& b = a.bp[p];
        const int gij = a.jobs[4 * job + 1];
        const int64_t cell = (int64_t)(gij & 0xFFFF) + (int64_t)(gij >> 16) * b.ny;
        // pairs that converged or have no further sweep, and masked cells, are skipped
        on = bp_live(b, a.it, a.done, p) && !(b.gmask && b.gmask[cell]);
        if (!on && a.rec && l == 0) a.rec[job] = __int_as_float(-1);  // no record for the epilogue
        const bool warped = a.it > 1 || b.has_pred0;
        A = warped ? b.warpA : b.A;
        B = warped ? b.warpB : b.B;
        M = b.mask;
        ld = b.nr;
      }
    }
    if (!__any_sync(FULL, on)) continue;
    // ---- the window's pixels into the plane, and their FP64 sums
    //      (load_windows!, src/correlators.jl:188-263; the mean is the exact
    //      sum over n rounded once)
    double sa = 0.0, sbb = 0.0;
    int cnt = 0;
    const int64_t base = (int64_t)rs + (int64_t)cs * ld + l;
    if (on) {
      constexpr int LB = W * C::CR < 16 ? W * C::CR : 16;
      static_assert(W * C::CR % LB == 0 && LB % C::CR == 0, "whole batches of whole columns");
      // batches of LB pixel pairs, all loads of a batch in flight before the
      // first is used (no branch between them)
#pragma unroll 1
      for (int i0 = 0; i0 < W * C::CR; i0 += LB) {
        float2 z[LB];
        uint32_t mk = 0u;
        const int64_t b0 = base + (int64_t)(i0 / C::CR) * ld;
#pragma unroll
        for (int i = 0; i < LB; ++i) {  // column (i0 + i) / CR, rows l + SEG (i % CR)
          const int64_t off = b0 + SEG * (i % C::CR) + (int64_t)(i / C::CR) * ld;
          z[i] = make_float2(ld_stream(A + off), ld_stream(B + off));
        }
        if (M) {
#pragma unroll
          for (int i = 0; i < LB; ++i)
            mk |= (uint32_t)(ld_stream(M + b0 + SEG * (i % C::CR) + (int64_t)(i / C::CR) * ld) != 0) << i;
        }
        cnt += LB - __popc(mk);
        float2* Pb = P + (i0 / C::CR) * LD + l;
#pragma unroll
        for (int i = 0; i < LB; ++i) {
          Pb[(i / C::CR) * LD + SEG * (i % C::CR)] = z[i];
          const bool m = mk >> i & 1u;  // a masked pixel leaves the mean
          sa += (double)(m ? 0.f : z[i].x);
          sbb += (double)(m ? 0.f : z[i].y);
        }
      }
    }
#pragma unroll
    for (int o = SEG / 2; o > 0; o >>= 1) {
      sa += __shfl_xor_sync(FULL, sa, o);
      sbb += __shfl_xor_sync(FULL, sbb, o);
      cnt += __shfl_xor_sync(FULL, cnt, o);
    }
    const bool bad = !(isfinite(sa) && isfinite(sbb));  // the window holds NaN or Inf
    const float ma = cnt > 0 && !bad ? (float)(sa / (double)cnt) : 0.f;
    const float mb = cnt > 0 && !bad ? (float)(sbb / (double)cnt) : 0.f;
    if (__any_sync(FULL, !on || bad || M)) {
      // a masked pixel takes the mean (it enters as ap * 0), a window that is
      // off or not finite is zero throughout
      for (int i = 0; i < W * C::CR; ++i) {
        const int p = SEG * (i % C::CR), q = i / C::CR;
        const bool z = !on || bad;
        if (z || (M && ld_stream(M + base + p + (int64_t)q * ld)))
          P[q * LD + p + l] = z ? make_float2(0.f, 0.f) : make_float2(ma, mb);
      }
    }
    __syncwarp();
    // ---- forward along p: the W data columns
#pragma unroll 1
    for (int j = 0; j < C::CR; ++j) {
      float2* L = P + (l + SEG * j) * LD;
      const float* ap = sap + (l + SEG * j) * (W + 1);
      float2 x[N];
#pragma unroll
      for (int p = 0; p < N; ++p) {
        x[p] = make_float2(0.f, 0.f);
        if (p < W) {
          const float2 z = L[p];
          // rounded here: not to be fused with the transform's first sums
          x[p] = make_float2(__fmul_rn(ap[p], __fsub_rn(z.x, ma)), __fmul_rn(ap[p], __fsub_rn(z.y, mb)));
        }
      }
      RDFT<N, false>::run(x, W);
#pragma unroll
      for (int k = 0; k < N; ++k) L[k] = x[k];
    }
    __syncwarp();
    // ---- forward along q, a row per lane, and the spectrum of its canonical
    //      columns q = 0 .. N/2. Rows of round j: HS j + (0 .. HS - 1) on the
    //      lower lanes and their negatives on the upper ones, but N/2 beside
    //      row 0 (both are their own negatives). Every lane overwrites only
    //      its own row.
#pragma unroll 1
    for (int j = 0; j < C::RR; ++j) {
      const int lh = l & (HS - 1);
      const bool self = j == 0 && lh == 0;
      const int p = l < HS ? HS * j + lh : (self ? H : N - HS * j - lh);
      const int partner = sb + (self ? l : l ^ HS);
      float2* L = P + p;
      float2 x[N];
#pragma unroll
      for (int q = 0; q < N; ++q) x[q] = q < W ? L[q * LD] : make_float2(0.f, 0.f);
      RDFT<N, false>::run(x, W);
      float2 S0 = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q <= H; ++q) {
        const float2 z = x[(N - q) % N];
        const float2 zm = make_float2(__shfl_sync(FULL, z.x, partner), __shfl_sync(FULL, z.y, partner));
        const float wk = PHASE ? ld_keep(a.phasew + q * N + p) : 1.f;
        const float2 S = cross_spectrum(x[q], zm, PHASE ? 1 : 0, wk);
        if (q == 0) S0 = S;
        else if (q < H) L[q * LD] = S;
        else L[0] = make_float2(S0.x - S.y, S0.y + S.x);  // columns 0 and N/2 as one
      }
    }
    __syncwarp();
    // ---- inverse along p: a canonical column per lane, the rows that hold a kept lag
    {
      float2* L = P + l * LD;
      float2 x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = L[k];
      RDFT<N, true>::run(x, N);
#pragma unroll
      for (int n = 0; n < N; ++n)
        if (C::keep(n)) L[n] = x[n];
    }
    __syncwarp();
    // ---- inverse along q of the row pair (blo + l, blo + l + nh) as
    //      T(p) + i T(p'), the normalised, gain-weighted magnitudes held until
    //      every lane has read its rows, then written as the real plane
    {
      float2 x[N];
      const bool act = l < nh, hasb = l + nh < nb;
      const int ps0 = blo + (act ? l : 0), ps1 = blo + (hasb ? l + nh : 0);
      const float2* La = P + (ps0 + H) % N;
      const float2* Lb = P + (ps1 + H) % N;
#pragma unroll
      for (int k = 0; k < H; ++k) {
        const float2 u = La[k * LD];
        const float2 v = hasb ? Lb[k * LD] : make_float2(0.f, 0.f);
        if (k == 0) {  // (column 0, column N/2), both real
          x[0] = make_float2(u.x, v.x);
          x[H] = make_float2(u.y, v.y);
        } else {
          x[k] = make_float2(u.x - v.y, u.y + v.x);
          x[N - k] = make_float2(u.x + v.y, v.x - u.y);
        }
      }
      RDFT<N, true>::run(x, N);
      float m0 = 0.f, m1 = 0.f;
      const float* g0 = s_gain + (ps0 - (H - Q));
      const float* g1 = s_gain + (hasb ? ps1 - (H - Q) : 0);
#pragma unroll
      for (int n = 0; n < N; ++n) {
        if (!C::keep(n)) continue;
        float r0 = fabsf(x[n].x) * scale, r1 = fabsf(x[n].y) * scale;
        if (C::BOXED) {
          r0 *= g0[(n + Q) % N * GB];
          r1 *= g1[(n + Q) % N * GB];
        }
        x[n] = make_float2(r0, r1);
        m0 = fmaxf(m0, r0);
        m1 = fmaxf(m1, r1);
      }
      if (!C::BOXED) {
        rmax[ps0] = __float_as_uint(m0);
        rmax[ps1] = __float_as_uint(m1);
      }
      __syncwarp();
      if (act) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
          if (!C::keep(n)) continue;
          const int qs = (n + H) % N;
          Rw[qs * LD + ps0] = x[n].x;
          if (!C::BOXED || hasb) Rw[qs * LD + ps1] = x[n].y;
        }
      }
    }
    __syncwarp();
    if (a.planes) {
      if (on) {
        float* dst = a.planes + job * (int64_t)(N * N);
        for (int e = l; e < N * N; e += SEG) {
          const int p = e % N, q = e / N;
          const bool in = !C::BOXED || (p >= blo && p <= bhi && q >= blo && q <= bhi);
          const float r = bad ? __int_as_float(0x7fc00000) : (in ? Rw[q * LD + p] : 0.f);
          dst[e] = a.accumulate ? dst[e] + r : r;
        }
      }
      if (a.accumulate) {  // ensemble planes are analysed once, after the last pair
        __syncwarp();
        continue;
      }
    }
    // ---- regional maxima and the peak record
    const bool scan = on && !bad;
    TopK<KC> tk;
    tk.init();
    if constexpr (C::BOXED) {
      for (int c0 = blo; c0 <= bhi; c0 += SEG) {  // a column of the box per lane
        const bool col = scan && c0 + l <= bhi;
        StripScan<true> st;
        st.init(Rw, LD, N, col ? c0 + l : blo, blo, col ? bhi + 1 : blo, blo, bhi, blo);
        constexpr int SU = 2;
        for (int r0 = blo; r0 <= bhi; r0 += SU) {
          float lb[SU], cb[SU], rb[SU];
          st.template load<SU>(r0, bhi + 1, lb, cb, rb);
#pragma unroll
          for (int u = 0; u < SU; ++u) st.step(r0 + u, lb[u], cb[u], rb[u], N, tk, K);
        }
      }
      // the last pixel, a zero among zeros (the only peak outside the box)
      if (scan && l == 0) tk.insert(fkey(0.f), ~(uint32_t)(N * N - 1), K);
    } else {
      seg_scan_rows<N>(tk, Rw, K, rmax, list, l, scan);
    }
    uint32_t mh, ml;
    const int nfound = seg_topk<SEG>(tk, K, l, mh, ml);
    if (l < nfound) {
      const int lin = (int)(~ml);
      s_vals[l] = __uint_as_float(mh & 0x7fffffffu);  // the key of a value >= 0 holds its bits
      s_locs[2 * l] = lin % N;
      s_locs[2 * l + 1] = lin / N;
    }
    __syncwarp();
    if (on)
      for (int wd = l; wd < nw; wd += SEG) {
        float val = 0.f;
        if (wd == 0) {
          val = __int_as_float(nfound);
        } else if (wd <= K) {
          if (wd - 1 < nfound) val = s_vals[wd - 1];
        } else if (wd <= 3 * K) {
          if ((wd - 1 - K) >> 1 < nfound) val = __int_as_float(s_locs[wd - 1 - K]);
        } else {
          const uint32_t e = s_map[wd];
          const int m = e & 0xff;
          if (m < nfound) {
            const int i = s_locs[2 * m] + (int)(e >> 8 & 0xff) - 2, j = s_locs[2 * m + 1] + (int)(e >> 16) - 2;
            if (i >= blo && i <= bhi && j >= blo && j <= bhi) val = Rw[j * LD + i];
          }
        }
        a.rec[(int64_t)wd * a.njobs + job] = val;
      }
    __syncwarp();  // the plane is reused by the warp's next windows
  }
}

template <int N, int W, int KC, bool PHASE> static cudaError_t launch_seg_k(const CorrArgs& a, cudaStream_t s, int num_sms) {
  using C = SegCfg<N, W>;
  const size_t sm = C::smem();
  if (C::BOXED && !(a.gain && a.box_hi > 0 && a.box_lo >= C::H - C::Q && a.box_hi <= C::H + C::Q))
    return cudaErrorInvalidValue;
  static DeviceOnce attr;
  cudaError_t e = raise_smem_carveout(attr, correlate_seg_kernel<N, W, KC, PHASE>, sm);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, correlate_seg_kernel<N, W, KC, PHASE>, C::NT, sm);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int64_t units = (a.njobs + C::WIN - 1) / C::WIN;
  int64_t grid = (int64_t)per_sm * num_sms;
  if (grid > units) grid = units;
  correlate_seg_kernel<N, W, KC, PHASE><<<(unsigned)grid, C::NT, sm, s>>>(a);
  e = cudaGetLastError();
  if (e == cudaSuccess && !a.accumulate) e = launch_peak_epilogue(a, N, s, num_sms);
  return e;
}

// regional maxima through the peak record, or planes summed without analysis
static inline bool seg_serves(const CorrArgs& a) { return a.accumulate || (a.rec && a.finder == 0); }
template <int N, int W> static cudaError_t launch_seg(const CorrArgs& a, cudaStream_t s, int num_sms) {
  if (a.method == 1)
    return a.npeaks <= 4 ? launch_seg_k<N, W, 4, true>(a, s, num_sms) : launch_seg_k<N, W, KMAX, true>(a, s, num_sms);
  return a.npeaks <= 4 ? launch_seg_k<N, W, 4, false>(a, s, num_sms) : launch_seg_k<N, W, KMAX, false>(a, s, num_sms);
}

}  // namespace hh
