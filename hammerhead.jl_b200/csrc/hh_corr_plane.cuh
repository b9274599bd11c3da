// General-shape window correlation with the plane in shared memory (sm_100a),
// included by k_correlate.cu.
//
// For the shapes of hh_corr_general.cuh (any FFT lengths with prime factors up
// to 61, rectangular windows and search areas) whose plane fits a CTA's shared
// memory twice. One CTA per window; every step runs over all lines of the
// plane at once, its butterflies dealt over the CTA's threads with the line
// index fastest: consecutive threads work on neighbouring lines, so every
// access is conflict-free (columns are NR|1 apart), twiddles are broadcast,
// and no lane idles because a line has fewer butterflies than a warp has
// lanes. The transforms are hh_corr_general.cuh's, value by value: Stockham
// stages of the same radices, and the 16 x B split for lengths 32, 64, 128 and
// 256, ping-pong between two planes. The first inverse stage forms the
// spectrum as it reads. CTAs have 128, 256 or 512 threads by the plane's size
// (gcorr_setup), up to 6, 2 or 1 of them to an SM.
// Bound by issue: a warp per line left 12 of 32 lanes busy in a 48-point
// radix-4 stage and 2 of 16 in the 16-point transforms of a 32-point line
// (63 k warp instructions per 48 x 32 plane, 21 k now). 8001 windows of
// 24 x 16 padded with the exclusion finder: 0.95 -> 0.33 ms; a 771 x 1030 pair
// with (48, 32), (24, 16) windows: correlation 2.0 -> 0.6 ms.
// (Included inside namespace hh, after hh_corr_general.cuh.)
#pragma once

// Lines of a batch: element e of line l at base[l * ls + e * es].
struct LineSet {
  int n;       // number of lines
  uint32_t inv;  // 2^32 / n + 1: k / n = umulhi(k, inv) for k n < 2^32
  int ls, es;
  __device__ __forceinline__ LineSet(int n_, int ls_, int es_) : n(n_), inv(0xffffffffu / n_ + 1u), ls(ls_), es(es_) {}
  // item k: line (fastest) and index within the line
  __device__ __forceinline__ void item(int k, int& l, int& i) const {
    i = n == 1 ? k : (int)__umulhi((uint32_t)k, inv);
    l = k - i * n;
  }
};

// A value as it would be stored: rounded here, so that the compiler does not
// fuse the products it comes from with the additions that use it (the planes
// then equal those of the kernel that passes it through memory).
__device__ __forceinline__ float2 rounded(float2 v) {
  asm("" : "+f"(v.x), "+f"(v.y));
  return v;
}

// x w (or x conj(w)) with the fused operations that hh_corr_general.cuh's
// products compile to
template <bool INV> __device__ __forceinline__ float2 cmul_fixed(float2 x, float2 w) {
  return INV ? make_float2(__fmaf_rn(x.x, w.x, __fmul_rn(x.y, w.y)), __fmaf_rn(x.y, w.x, -__fmul_rn(x.x, w.y)))
             : make_float2(__fmaf_rn(x.x, w.x, -__fmul_rn(x.y, w.y)), __fmaf_rn(x.x, w.y, __fmul_rn(x.y, w.x)));
}

// One Stockham stage of compile-time radix R over a set of lines (gc_stage's
// arithmetic): get(l, e) reads element e of line l, put(l, e, v) writes it;
// p the product of the radices before, nr = n / R, tstep = n / (p R).
template <int R, bool INV, class Get, class Put>
__device__ __forceinline__ void pl_stage(const LineSet& L, int p, int nr, int tstep, const float2* tw, int tid, int nt,
                                         const Get& get, const Put& put) {
  const bool pow2 = (p & (p - 1)) == 0;
  for (int it = tid; it < L.n * nr; it += nt) {
    int l, i;
    L.item(it, l, i);
    const int k = pow2 ? (i & (p - 1)) : i % p, j0 = (i - k) * R + k;
    float2 x[R];
#pragma unroll
    for (int m = 0; m < R; ++m) x[m] = rounded(get(l, i + m * nr));
    if (k) {
#pragma unroll
      for (int m = 1; m < R; ++m) x[m] = cmul_fixed<INV>(x[m], tw[m * k * tstep]);
    }
    if constexpr (R == 2) {
      put(l, j0, make_float2(x[0].x + x[1].x, x[0].y + x[1].y));
      put(l, j0 + p, make_float2(x[0].x - x[1].x, x[0].y - x[1].y));
    } else if constexpr (R == 4) {
      const float2 a = make_float2(x[0].x + x[2].x, x[0].y + x[2].y), b = make_float2(x[0].x - x[2].x, x[0].y - x[2].y);
      const float2 c = make_float2(x[1].x + x[3].x, x[1].y + x[3].y), d = make_float2(x[1].x - x[3].x, x[1].y - x[3].y);
      const float2 md = INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);  // -+ i d
      put(l, j0, make_float2(a.x + c.x, a.y + c.y));
      put(l, j0 + p, make_float2(b.x + md.x, b.y + md.y));
      put(l, j0 + 2 * p, make_float2(a.x - c.x, a.y - c.y));
      put(l, j0 + 3 * p, make_float2(b.x - md.x, b.y - md.y));
    } else {
      float2 w[R];
#pragma unroll
      for (int e = 1; e < R; ++e) w[e] = tw[e * nr];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int m = 0; m < R; ++m) {
          const float2 v = (m * q) % R ? cmul_fixed<INV>(x[m], w[(m * q) % R]) : x[m];
          acc.x += v.x;
          acc.y += v.y;
        }
        put(l, j0 + q * p, acc);
      }
    }
  }
}
// The same for a run-time radix (11 and above): an item per output, its inputs
// read again. (An item per butterfly left 14 threads of a CTA with all of a 14 x
// 41 plane's 41-point rows: 396 us for up to 440 windows, 76 to 85 now.)
template <bool INV, class Get, class Put>
__device__ __forceinline__ void pl_stage_any(const LineSet& L, int r, int p, int nr, int tstep, const float2* tw, int tid,
                                             int nt, const Get& get, const Put& put) {
  for (int it = tid; it < L.n * nr * r; it += nt) {
    int l, iq;
    L.item(it, l, iq);
    const int q = iq / nr, i = iq - q * nr, k = i % p, j0 = (i - k) * r + k;
    float2 acc = make_float2(0.f, 0.f);
    int e = 0;
    for (int m = 0; m < r; ++m) {
      float2 x = rounded(get(l, i + m * nr));
      if (k && m) x = cmul_fixed<INV>(x, tw[m * k * tstep]);
      if (e) x = cmul_fixed<INV>(x, tw[e * nr]);
      acc.x += x.x;
      acc.y += x.y;
      e += q;
      if (e >= r) e -= r;
    }
    put(l, j0 + q * p, acc);
  }
}

// Lengths 16 B: the 16-point transforms over n1 with the twiddle (first step,
// result at index k1 B + n2) and the B-point ones over n2 (second step).
template <int B, bool INV, class Get, class Put>
__device__ __forceinline__ void pl_first16(const LineSet& L, const float2* tw, int tid, int nt, const Get& get,
                                           const Put& put) {
  for (int it = tid; it < L.n * B; it += nt) {
    int l, n2;
    L.item(it, l, n2);
    float2 x[16];
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) x[n1] = rounded(get(l, B * n1 + n2));
    RDFT<16, INV>::run(x, 16);
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) {
      float2 v = x[k1];
      if (k1 && n2) v = cmul_fixed<INV>(v, tw[n2 * k1]);
      put(l, k1 * B + n2, v);
    }
  }
}
template <int B, bool INV, class Get, class Put>
__device__ __forceinline__ void pl_second16(const LineSet& L, int tid, int nt, const Get& get, const Put& put) {
  for (int it = tid; it < L.n * 16; it += nt) {
    int l, k1;
    L.item(it, l, k1);
    float2 t[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) t[n2] = get(l, k1 * B + n2);
    RDFT<B, INV>::run(t, B);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) put(l, k1 + 16 * k2, t[k2]);
  }
}

// Length-n transform of a set of lines: `first` reads the inputs, the stages
// go back and forth between the two planes (src = which of them holds the
// inputs; the first stage writes the other), `keep(l, e)` says whether the
// last stage stores element e. Returns the plane that holds the result.
// Every stage ends with a CTA barrier.
template <bool INV, class First, class Keep>
__device__ __forceinline__ int pl_lines(float2* Z0, float2* Z1, int src, const LineSet& L, int n, const int8_t* radix,
                                        int nst, const float2* tw, int tid, int nt, const First& first, const Keep& keep) {
  const int ls = L.ls, es = L.es;
  auto plane = [&](int w) { return w ? Z1 : Z0; };
  if (gc_reg_len(n)) {
    float2* o1 = plane(src ^ 1);
    float2* o2 = plane(src);
    const int B = n / 16;
    auto put1 = [&](int l, int e, float2 v) { o1[l * ls + e * es] = v; };
    auto get2 = [&](int l, int e) { return o1[l * ls + e * es]; };
    auto put2 = [&](int l, int e, float2 v) {
      if (keep(l, e)) o2[l * ls + e * es] = v;
    };
#define X(b)                                              \
  if (B == b) {                                           \
    pl_first16<b, INV>(L, tw, tid, nt, first, put1);      \
    __syncthreads();                                      \
    pl_second16<b, INV>(L, tid, nt, get2, put2);          \
  }
    X(2) else X(4) else X(8) else X(16)
#undef X
    __syncthreads();
    return src;
  }
  int p = 1;
  for (int s = 0; s < nst; ++s) {
    const int r = radix[s], nr = n / r, tstep = nr / p;
    const float2* in = plane(src);
    float2* out = plane(src ^ 1);
    const bool f = s == 0, lastst = s == nst - 1;
    auto get = [&](int l, int e) { return f ? first(l, e) : in[l * ls + e * es]; };
    auto put = [&](int l, int e, float2 v) {
      if (!lastst || keep(l, e)) out[l * ls + e * es] = v;
    };
    switch (r) {
      case 2: pl_stage<2, INV>(L, p, nr, tstep, tw, tid, nt, get, put); break;
      case 3: pl_stage<3, INV>(L, p, nr, tstep, tw, tid, nt, get, put); break;
      case 4: pl_stage<4, INV>(L, p, nr, tstep, tw, tid, nt, get, put); break;
      case 5: pl_stage<5, INV>(L, p, nr, tstep, tw, tid, nt, get, put); break;
      case 7: pl_stage<7, INV>(L, p, nr, tstep, tw, tid, nt, get, put); break;
      default: pl_stage_any<INV>(L, r, p, nr, tstep, tw, tid, nt, get, put);
    }
    __syncthreads();
    p *= r;
    src ^= 1;
  }
  return src;
}

// shared memory: two planes, the real box, the twiddle tables, the reduction
// and peak slots
__host__ __device__ inline size_t plane_smem(int NR, int NC, int nboxr, int nboxc, int warps) {
  return 2 * (size_t)NC * (NR | 1) * sizeof(float2) + (size_t)(NR + NC) * sizeof(float2) +
         (((size_t)nboxc * (nboxr | 1) + 3) & ~(size_t)3) * sizeof(float) + gcorr_smem_extra(warps);
}

// CTAs of 128 threads per SM that the registers are sized for
constexpr int PLANE_CTAS = gcorr_plane_ctas;

template <int THREADS, bool BOXED>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? PLANE_CTAS : 512 / THREADS) correlate_plane_kernel(const CorrArgs a) {
  constexpr int WARPS = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int NR = a.nfr, NC = a.nfc, wr = a.wr, wc = a.wc, sr = a.sr, sc = a.sc;
  const int ldz = NR | 1;
  const int rlo = a.gc_box[0], rhi = a.gc_box[1], clo = a.gc_box[2], chi = a.gc_box[3];
  const int nboxr = rhi - rlo + 1, nboxc = chi - clo + 1, ldb = nboxr | 1;
  float2* Z0 = reinterpret_cast<float2*>(smem_raw);
  float2* Z1 = Z0 + NC * ldz;
  float2* twr = Z1 + NC * ldz;
  float2* twc = twr + NR;
  float* Rb = reinterpret_cast<float*>(twc + NC);
  float* R = Rb - (clo * ldb + rlo);  // column js at js * ldb, row is (both fftshifted)
  double* part = reinterpret_cast<double*>(Rb + ((nboxc * ldb + 3) & ~3));  // WARPS x 4
  uint32_t* red = reinterpret_cast<uint32_t*>(part + 4 * WARPS);
  float* s_vals = reinterpret_cast<float*>(red + WARPS * 2 * KMAX);
  int* s_locs = reinterpret_cast<int*>(s_vals + KMAX);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = a.npeaks > 2 ? a.npeaks : 2;
  const int64_t P = (int64_t)NR * NC;
  const int oar = (sr - wr) / 2, oac = (sc - wc) / 2;  // frame-A window inside the search area
  const bool search = sr != wr || sc != wc;
  const float scale = 1.0f / (float)P;
  const ScanPlan sp = scan_plan(tid, THREADS, rlo, rhi, clo, chi);
  PeakOut po{a.du, a.dv, a.ratio, a.moment, a.alt_u, a.alt_v, a.nalt, a.G, a.packed, a.locs};
  for (int k = tid; k < NR; k += THREADS) twr[k] = a.twr[k];
  for (int k = tid; k < NC; k += THREADS) twc[k] = a.twc[k];
  __syncthreads();
  const LineSet pix(sr, 0, 0);  // items (row fastest, column)
  auto all = [](int, int) { return true; };

  for (int64_t job = blockIdx.x; job < a.njobs; job += gridDim.x) {
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
      if (!bp_live(b, a.it, a.done, p) || (b.gmask && b.gmask[cell])) continue;  // uniform across the CTA
      const bool warped = a.it > 1 || b.has_pred0;
      A = warped ? b.warpA : b.A;
      B = warped ? b.warpB : b.B;
      M = b.mask;
      ld = b.nr;
      gid = b.goff + cell;
      pw.G = (int64_t)b.ny * b.nx;
      pw.nalt = b.nalt;
      pw.alt_u = a.alt_u ? a.alt_u + b.aoff - b.goff : nullptr;
      pw.alt_v = a.alt_v ? a.alt_v + b.aoff - b.goff : nullptr;
    } else {
      gid = (int64_t)a.jobs[4 * job] + (int64_t)a.jobs[4 * job + 1] * a.ny;
    }
    // search-area origin: the window's origin less the centring offset
    const int64_t w0 = (int64_t)a.jobs[4 * job + 2] - oar + ((int64_t)a.jobs[4 * job + 3] - oac) * ld;

    // ---- the pixels into plane 0 (frame A outside its window 0), and the
    //      means over the unmasked ones (FP64, one rounding)
    double sa = 0.0, sb = 0.0;
    int na = 0, nb = 0;
    for (int k0 = tid; k0 < sr * sc; k0 += 4 * THREADS) {
      float va[4], vb[4];
      bool mk[4], ina[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u * THREADS;
        const bool in = k < sr * sc;
        int i, j;
        pix.item(in ? k : 0, i, j);
        ina[u] = in && (unsigned)(i - oar) < (unsigned)wr && (unsigned)(j - oac) < (unsigned)wc;
        const int64_t off = w0 + i + j * ld;
        va[u] = ld_stream_if(A + off, ina[u]);
        vb[u] = ld_stream_if(B + off, in);
        mk[u] = !in || ld_stream_if(M + off, in && M) != 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u * THREADS;
        sb += (double)(mk[u] ? 0.f : vb[u]);
        sa += (double)(mk[u] ? 0.f : va[u]);
        nb += !mk[u];
        na += ina[u] && !mk[u];
        if (k < sr * sc) {
          int i, j;
          pix.item(k, i, j);
          Z0[j * ldz + i] = make_float2(va[u], vb[u]);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sa += __shfl_xor_sync(0xffffffffu, sa, o);
      sb += __shfl_xor_sync(0xffffffffu, sb, o);
    }
    na = __reduce_add_sync(0xffffffffu, na);
    nb = __reduce_add_sync(0xffffffffu, nb);
    if (lane == 0) {
      part[4 * warp] = sa;
      part[4 * warp + 1] = sb;
      part[4 * warp + 2] = (double)na;
      part[4 * warp + 3] = (double)nb;
    }
    __syncthreads();
    double ta = 0.0, tb = 0.0, tna = 0.0, tnb = 0.0;
    for (int w = 0; w < WARPS; ++w) {
      ta += part[4 * w];
      tb += part[4 * w + 1];
      tna += part[4 * w + 2];
      tnb += part[4 * w + 3];
    }
    const float ma = tna > 0 ? (float)(ta / tna) : 0.f, mb = tnb > 0 ? (float)(tb / tnb) : 0.f;
    const bool bad = !(isfinite(ta) && isfinite(tb));  // the window holds NaN or Inf: the reference's plane is NaN
    // ---- mean and apodization (load_windows!); masked pixels are zero in both
    for (int k = tid; k < sr * sc; k += THREADS) {
      int i, j;
      pix.item(k, i, j);
      const int ia = i - oar, ja = j - oac;
      const bool ina = (unsigned)ia < (unsigned)wr && (unsigned)ja < (unsigned)wc;
      const bool on = !bad && !ld_stream_if(M + w0 + i + j * ld, M != nullptr);
      const float ap = ld_keep_if(a.apod + ia + ja * wr, ina);
      float2* c = Z0 + j * ldz + i;
      const float2 z = *c;
      float2 v = make_float2(0.f, 0.f);
      if (on) {
        if (ina) v.x = __fmul_rn(ap, __fsub_rn(z.x, ma));
        v.y = search ? __fsub_rn(z.y, mb) : __fmul_rn(ap, __fsub_rn(z.y, mb));
      }
      *c = v;
    }
    __syncthreads();

    // ---- forward: the data columns, then every row
    int at = pl_lines<false>(
        Z0, Z1, 0, LineSet(sc, ldz, 1), NR, a.gc_radix_r, a.gc_nst_r, twr, tid, THREADS,
        [&](int l, int e) { return e < sr ? Z0[l * ldz + e] : make_float2(0.f, 0.f); }, all);
    {
      const float2* Zc = at ? Z1 : Z0;
      at = pl_lines<false>(
          Z0, Z1, at, LineSet(NR, 1, ldz), NC, a.gc_radix_c, a.gc_nst_c, twc, tid, THREADS,
          [&](int l, int e) { return e < sc ? Zc[e * ldz + l] : make_float2(0.f, 0.f); }, all);
    }
    // ---- the spectrum from Z(k) and Z(-k), inverse along the rows; the
    //      box's columns are kept
    {
      const float2* Zf = at ? Z1 : Z0;
      at = pl_lines<true>(
          Z0, Z1, at, LineSet(NR, 1, ldz), NC, a.gc_radix_c, a.gc_nst_c, twc, tid, THREADS,
          [&](int l, int e) {
            const int lm = l == 0 ? 0 : NR - l, em = e == 0 ? 0 : NC - e;
            const float wk = a.phasew ? __ldg(a.phasew + l + (int64_t)e * NR) : 1.f;
            return cross_spectrum(Zf[e * ldz + l], Zf[em * ldz + lm], a.method, wk);
          },
          [&](int, int e) {
            const int js = e + NC / 2 < NC ? e + NC / 2 : e + NC / 2 - NC;
            return js >= clo && js <= chi;
          });
    }
    // ---- the box's columns back: line b is the fftshifted column clo + b
    {
      const float2* Zr = at ? Z1 : Z0;
      at = pl_lines<true>(
          Z0, Z1, at, LineSet(nboxc, ldz, 1), NR, a.gc_radix_r, a.gc_nst_r, twr, tid, THREADS,
          [&](int l, int e) {
            const int js = clo + l, j = js >= NC / 2 ? js - NC / 2 : js - NC / 2 + NC;
            return Zr[j * ldz + e];
          },
          all);
    }
    // ---- |.| / (nr nc), fftshift, gain, for the box
    {
      const float2* Zr = at ? Z1 : Z0;
      const LineSet box(nboxr, 0, 0);
      for (int k = tid; k < nboxr * nboxc; k += THREADS) {
        int i, b;
        box.item(k, i, b);
        const int is = rlo + i, js = clo + b;
        const float2 c = Zr[b * ldz + (is >= NR / 2 ? is - NR / 2 : is - NR / 2 + NR)];
        float v = hypotf(c.x * scale, c.y * scale);
        if (a.gain) v *= __ldg(a.gain + is + (int64_t)js * NR);
        if (bad) v = __int_as_float(0x7fc00000);
        R[js * ldb + is] = v;
      }
    }
    __syncthreads();
    // ---- plane out (correlation_planes / ensemble sums) and analysis
    if (a.planes) {  // a window holding NaN or Inf has a NaN plane, as in the reference
      float* dst = a.planes + job * P;
      const LineSet rows(NR, 0, 0);
      for (int e = tid; e < NR * NC; e += THREADS) {
        int is, js;
        rows.item(e, is, js);
        const bool in = !BOXED || (is >= rlo && is <= rhi && js >= clo && js <= chi);
        const float v = bad ? __int_as_float(0x7fc00000) : (in ? R[js * ldb + is] : 0.f);
        dst[e] = a.accumulate ? dst[e] + v : v;
      }
    }
    if (!a.accumulate)
      analyze_group<0, BOXED>(R, NR, NC, ldb, K, a.npeaks, a.finder, a.subpixel, tid, THREADS, red, true, s_vals, s_locs,
                              gid, job, &pw, bad, 0, sp, nullptr, 0);
    __syncthreads();  // the planes and shared buffers are reused by the CTA's next window
  }
}

template <int THREADS, bool BOXED> static cudaError_t launch_plane(const CorrArgs& a, cudaStream_t s) {
  // raised to the device's limit at once: launches of different shapes may share a graph
  static DeviceOnce attr;
  const cudaError_t e = raise_smem(attr, correlate_plane_kernel<THREADS, BOXED>, 227 * 1024);
  if (e != cudaSuccess) return e;
  const int64_t grid = a.njobs < a.gscr_slices ? a.njobs : a.gscr_slices;
  correlate_plane_kernel<THREADS, BOXED><<<(unsigned)grid, THREADS, a.gc_smem_bytes, s>>>(a);
  return cudaGetLastError();
}
