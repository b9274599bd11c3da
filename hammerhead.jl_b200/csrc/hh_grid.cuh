// Per-cell operations on a column-major (ny, nx) vector grid, shared by the
// single-pair kernels (k_vector.cu) and the batched ones (k_batch.cu). Each
// restates src/quality.jl / src/pipeline.jl in the reference's precision
// (Float32 fields, Float64 where Julia widens) with explicit round-to-nearest
// arithmetic, so flags and replaced values equal the CPU restatement bit for
// bit on identical inputs. Pointers address the grid of one image pair.
#pragma once
#include <cooperative_groups.h>
#include <math.h>
#include <stdint.h>

namespace hh {

#define FADD(a, b) __fadd_rn((a), (b))
#define FSUB(a, b) __fsub_rn((a), (b))
#define FMUL(a, b) __fmul_rn((a), (b))

static __device__ __forceinline__ float f_nan() { return __int_as_float(0x7fc00000); }

// Statistics.median! on a small local array: NaN if any NaN; even n ->
// a/2 + b/2 of the two middle order statistics.
template <class T> __device__ __forceinline__ void isort(T* a, int n) {
  for (int i = 1; i < n; ++i) {
    T x = a[i];
    int j = i - 1;
    while (j >= 0 && a[j] > x) {
      a[j + 1] = a[j];
      --j;
    }
    a[j + 1] = x;
  }
}
__device__ __forceinline__ float median_f(float* a, int n) {
  for (int i = 0; i < n; ++i)
    if (isnan(a[i])) return f_nan();
  isort(a, n);
  if (n & 1) return a[n / 2];
  return FADD(a[n / 2 - 1] / 2.0f, a[n / 2] / 2.0f);
}
__device__ __forceinline__ double median_d(double* a, int n) {
  for (int i = 0; i < n; ++i)
    if (isnan(a[i])) return __longlong_as_double(0x7ff8000000000000LL);
  isort(a, n);
  if (n & 1) return a[n / 2];
  return __dadd_rn(a[n / 2 - 1] / 2.0, a[n / 2] / 2.0);
}

constexpr int UOD_MAXN = 80;  // neighbourhood <= 4 layers


// Neighbourhoods of 1 and 2 layers in registers: the S = (2nb+1)^2 - 1
// neighbour slots hold +inf where a neighbour is missing (edge or excluded),
// so sorting the slots with a fixed comparator network puts the n present
// values first, in order, and no array needs dynamic indexing. The networks
// are Batcher's odd-even merge sort (19 comparators for 8 inputs; the
// 32-input network without the comparators that reach slots 24..31, which
// hold +inf throughout, for 24); both sort every 0/1 input (checked
// exhaustively), hence every input. The medians equal median_f's up to the
// sign of a zero, which only ever enters through |x - m|.
__device__ __forceinline__ void cas(float& a, float& b) {
  const float lo = fminf(a, b), hi = fmaxf(a, b);
  a = lo;
  b = hi;
}
__device__ __forceinline__ void cas(double& a, double& b) {
  const bool swap = a > b;
  const double lo = swap ? b : a, hi = swap ? a : b;
  a = lo;
  b = hi;
}
template <class T> __device__ __forceinline__ void sort_net(T (&a)[8]) {
  cas(a[0], a[1]); cas(a[2], a[3]); cas(a[4], a[5]); cas(a[6], a[7]); cas(a[0], a[2]); cas(a[1], a[3]);
  cas(a[4], a[6]); cas(a[5], a[7]); cas(a[1], a[2]); cas(a[5], a[6]); cas(a[0], a[4]); cas(a[3], a[7]);
  cas(a[1], a[5]); cas(a[2], a[6]); cas(a[1], a[4]); cas(a[3], a[6]); cas(a[2], a[4]); cas(a[3], a[5]);
  cas(a[3], a[4]);
}
template <class T> __device__ __forceinline__ void sort_net(T (&a)[24]) {
  cas(a[0], a[1]); cas(a[2], a[3]); cas(a[0], a[2]); cas(a[1], a[3]); cas(a[1], a[2]); cas(a[4], a[5]);
  cas(a[6], a[7]); cas(a[4], a[6]); cas(a[5], a[7]); cas(a[5], a[6]); cas(a[0], a[4]); cas(a[2], a[6]);
  cas(a[2], a[4]); cas(a[1], a[5]); cas(a[3], a[7]); cas(a[3], a[5]); cas(a[1], a[2]); cas(a[3], a[4]);
  cas(a[5], a[6]); cas(a[8], a[9]); cas(a[10], a[11]); cas(a[8], a[10]); cas(a[9], a[11]); cas(a[9], a[10]);
  cas(a[12], a[13]); cas(a[14], a[15]); cas(a[12], a[14]); cas(a[13], a[15]); cas(a[13], a[14]); cas(a[8], a[12]);
  cas(a[10], a[14]); cas(a[10], a[12]); cas(a[9], a[13]); cas(a[11], a[15]); cas(a[11], a[13]); cas(a[9], a[10]);
  cas(a[11], a[12]); cas(a[13], a[14]); cas(a[0], a[8]); cas(a[4], a[12]); cas(a[4], a[8]); cas(a[2], a[10]);
  cas(a[6], a[14]); cas(a[6], a[10]); cas(a[2], a[4]); cas(a[6], a[8]); cas(a[10], a[12]); cas(a[1], a[9]);
  cas(a[5], a[13]); cas(a[5], a[9]); cas(a[3], a[11]); cas(a[7], a[15]); cas(a[7], a[11]); cas(a[3], a[5]);
  cas(a[7], a[9]); cas(a[11], a[13]); cas(a[1], a[2]); cas(a[3], a[4]); cas(a[5], a[6]); cas(a[7], a[8]);
  cas(a[9], a[10]); cas(a[11], a[12]); cas(a[13], a[14]); cas(a[16], a[17]); cas(a[18], a[19]); cas(a[16], a[18]);
  cas(a[17], a[19]); cas(a[17], a[18]); cas(a[20], a[21]); cas(a[22], a[23]); cas(a[20], a[22]); cas(a[21], a[23]);
  cas(a[21], a[22]); cas(a[16], a[20]); cas(a[18], a[22]); cas(a[18], a[20]); cas(a[17], a[21]); cas(a[19], a[23]);
  cas(a[19], a[21]); cas(a[17], a[18]); cas(a[19], a[20]); cas(a[21], a[22]); cas(a[18], a[20]); cas(a[19], a[21]);
  cas(a[17], a[18]); cas(a[19], a[20]); cas(a[21], a[22]); cas(a[0], a[16]); cas(a[8], a[16]); cas(a[4], a[20]);
  cas(a[12], a[20]); cas(a[4], a[8]); cas(a[12], a[16]); cas(a[2], a[18]); cas(a[10], a[18]); cas(a[6], a[22]);
  cas(a[14], a[22]); cas(a[6], a[10]); cas(a[14], a[18]); cas(a[2], a[4]); cas(a[6], a[8]); cas(a[10], a[12]);
  cas(a[14], a[16]); cas(a[18], a[20]); cas(a[1], a[17]); cas(a[9], a[17]); cas(a[5], a[21]); cas(a[13], a[21]);
  cas(a[5], a[9]); cas(a[13], a[17]); cas(a[3], a[19]); cas(a[11], a[19]); cas(a[7], a[23]); cas(a[15], a[23]);
  cas(a[7], a[11]); cas(a[15], a[19]); cas(a[3], a[5]); cas(a[7], a[9]); cas(a[11], a[13]); cas(a[15], a[17]);
  cas(a[19], a[21]); cas(a[1], a[2]); cas(a[3], a[4]); cas(a[5], a[6]); cas(a[7], a[8]); cas(a[9], a[10]);
  cas(a[11], a[12]); cas(a[13], a[14]); cas(a[15], a[16]); cas(a[17], a[18]); cas(a[19], a[20]); cas(a[21], a[22]);
}

// sorts the slots and returns the two middle order statistics of the n (1..S)
// present ones; false when one of them is NaN
template <int S, class T> __device__ __forceinline__ bool middle_net(T (&a)[S], int n, T& lo, T& hi) {
  bool nan = false;
#pragma unroll
  for (int i = 0; i < S; ++i) nan |= isnan(a[i]);
  if (nan) return false;
  sort_net(a);
  const int h = n / 2;
  lo = hi = a[0];  // a[h - 1], a[h]
#pragma unroll
  for (int i = 1; i < S; ++i) {
    if (i == h) hi = a[i];
    if (i == h - 1) lo = a[i];
  }
  return true;
}
template <int S> __device__ __forceinline__ float median_net_f(float (&a)[S], int n) {
  float lo, hi;
  if (!middle_net(a, n, lo, hi)) return f_nan();
  if (n & 1) return hi;
  return FADD(lo / 2.0f, hi / 2.0f);
}
// median_d of the present slots: floats are sorted as floats, which orders
// them like their doubles
template <int S, class T> __device__ __forceinline__ double median_net_d(T (&a)[S], int n) {
  T lo, hi;
  if (!middle_net(a, n, lo, hi)) return __longlong_as_double(0x7ff8000000000000LL);
  if (n & 1) return (double)hi;
  return __dadd_rn((double)lo / 2.0, (double)hi / 2.0);
}

// The slots of cell (r, c): bit s of near_present is set where neighbour s is
// on the grid and neither flagged nor masked (either may be null). Slots off
// the grid read the flags of the nearest cell on it, so that no load waits
// behind a branch: a test per neighbour serialises the S loads of each array
// (1.5 ms for the substitutions of the series below, against 1.2).
template <int NB> __device__ __forceinline__ bool near_on(int ny, int nx, int r, int c, int s, int64_t& q) {
  constexpr int D = 2 * NB + 1, S = D * D - 1;
  const int d = s < S / 2 ? s : s + 1;  // skip the centre of the D x D block
  const int r2 = r + d % D - NB, c2 = c + d / D - NB;
  const int r3 = min(max(r2, 0), ny - 1), c3 = min(max(c2, 0), nx - 1);
  q = r3 + (int64_t)c3 * ny;
  return r2 == r3 && c2 == c3;
}
template <int NB>
__device__ __forceinline__ uint32_t near_present(int ny, int nx, int r, int c, const uint8_t* flags,
                                                 const uint8_t* gmask) {
  constexpr int D = 2 * NB + 1, S = D * D - 1;
  uint32_t on = 0, off = 0;
  int64_t q;
#pragma unroll
  for (int s = 0; s < S; ++s) on |= near_on<NB>(ny, nx, r, c, s, q) ? 1u << s : 0u;
  if (flags) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      near_on<NB>(ny, nx, r, c, s, q);
      off |= flags[q] ? 1u << s : 0u;
    }
  }
  if (gmask) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      near_on<NB>(ny, nx, r, c, s, q);
      off |= gmask[q] ? 1u << s : 0u;
    }
  }
  return on & ~off;
}
// *p where `on`, else +inf, as one predicated load: no branch between the loads
// of a neighbourhood, and no read of a neighbour that does not count, which
// another thread of the launch may be writing (a cell that counts keeps its
// value throughout the launch, so the compiler may place the load freely)
__device__ __forceinline__ float ld_present(const float* p, bool on) {
  float v;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.f32 %0, 0f7F800000;\n\t@p ld.global.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"((int)on));
  return v;
}
template <int NB, int S>
__device__ __forceinline__ void near_values(const float* f, int ny, int nx, int r, int c, uint32_t present,
                                            float (&x)[S]) {
  static_assert(S == (2 * NB + 1) * (2 * NB + 1) - 1, "");
#pragma unroll
  for (int s = 0; s < S; ++s) {
    int64_t q;
    near_on<NB>(ny, nx, r, c, s, q);
    x[s] = ld_present(f + q, (present >> s) & 1u);
  }
}

template <int NB>
__device__ __forceinline__ uint8_t uod_cell_net(const float* u, const float* v, int ny, int nx, int r, int c, double thr,
                                                double eps, const uint8_t* exclude) {
  constexpr int D = 2 * NB + 1, S = D * D - 1;
  const int64_t k = r + (int64_t)c * ny;
  const float INF = __int_as_float(0x7f800000);
  float nu[S], nv[S];
  uint32_t present = 0;
  int n = 0;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const int d = s < S / 2 ? s : s + 1;  // skip the centre of the D x D block
    const int r2 = r + d % D - NB, c2 = c + d / D - NB;
    const int64_t q = r2 + (int64_t)c2 * ny;
    const bool ok = r2 >= 0 && r2 < ny && c2 >= 0 && c2 < nx && !(exclude && exclude[q]);
    nu[s] = ok ? u[q] : INF;
    nv[s] = ok ? v[q] : INF;
    present |= ok ? 1u << s : 0u;
    n += ok;
  }
  if (n == 0) return 0;
  float ru[S], rv[S];
#pragma unroll
  for (int s = 0; s < S; ++s) {
    ru[s] = nu[s];
    rv[s] = nv[s];
  }
  const float um = median_net_f<S>(ru, n), vm = median_net_f<S>(rv, n);
#pragma unroll
  for (int s = 0; s < S; ++s) {
    const bool ok = (present >> s) & 1u;
    ru[s] = ok ? fabsf(FSUB(nu[s], um)) : INF;
    rv[s] = ok ? fabsf(FSUB(nv[s], vm)) : INF;
  }
  const double un = (double)fabsf(FSUB(u[k], um)) / __dadd_rn((double)median_net_f<S>(ru, n), eps);
  const double vn = (double)fabsf(FSUB(v[k], vm)) / __dadd_rn((double)median_net_f<S>(rv, n), eps);
  return (un > thr || vn > thr) ? 1 : 0;
}

// universal_outlier_detection (src/quality.jl:244-293) at cell (r, c).
__device__ __forceinline__ uint8_t uod_cell(const float* u, const float* v, int ny, int nx, int r, int c, double thr,
                                            int nb, double eps, const uint8_t* exclude) {
  const int64_t k = r + (int64_t)c * ny;
  if (exclude && exclude[k]) return 0;
  if (nb == 1) return uod_cell_net<1>(u, v, ny, nx, r, c, thr, eps, exclude);
  if (nb == 2) return uod_cell_net<2>(u, v, ny, nx, r, c, thr, eps, exclude);
  float nu[UOD_MAXN], nv[UOD_MAXN], ru[UOD_MAXN], rv[UOD_MAXN];
  int n = 0;
  for (int c2 = max(0, c - nb); c2 <= min(nx - 1, c + nb); ++c2)
    for (int r2 = max(0, r - nb); r2 <= min(ny - 1, r + nb); ++r2) {
      if (r2 == r && c2 == c) continue;
      const int64_t q = r2 + (int64_t)c2 * ny;
      if (exclude && exclude[q]) continue;
      nu[n] = u[q];
      nv[n] = v[q];
      ++n;
    }
  if (n == 0) return 0;
  for (int i = 0; i < n; ++i) {
    ru[i] = nu[i];
    rv[i] = nv[i];
  }
  const float um = median_f(ru, n), vm = median_f(rv, n);
  for (int i = 0; i < n; ++i) {
    ru[i] = fabsf(FSUB(nu[i], um));
    rv[i] = fabsf(FSUB(nv[i], vm));
  }
  const double un = (double)fabsf(FSUB(u[k], um)) / __dadd_rn((double)median_f(ru, n), eps);
  const double vn = (double)fabsf(FSUB(v[k], vm)) / __dadd_rn((double)median_f(rv, n), eps);
  return (un > thr || vn > thr) ? 1 : 0;
}

// Median of the n neighbours x[] of one field and the median absolute
// deviation from it, in double.
template <int S>
__device__ __forceinline__ void near_mad(const float (&x)[S], uint32_t present, int n, double& m, double& mad) {
  float t[S];
#pragma unroll
  for (int s = 0; s < S; ++s) t[s] = x[s];
  m = median_net_d(t, n);
  double d[S];
#pragma unroll
  for (int s = 0; s < S; ++s)
    d[s] = (present >> s) & 1u ? fabs(__dsub_rn((double)x[s], m)) : __longlong_as_double(0x7ff0000000000000LL);
  mad = median_net_d(d, n);
}
template <int NB>
__device__ __forceinline__ bool near_spread(const float* u, const float* v, int ny, int nx, int r, int c,
                                            const uint8_t* flags, const uint8_t* gmask, double& mu, double& mv,
                                            double& madu, double& madv) {
  constexpr int S = (2 * NB + 1) * (2 * NB + 1) - 1;
  const uint32_t present = near_present<NB>(ny, nx, r, c, flags, gmask);
  const int n = __popc(present);
  if (n < 3) return false;
  float x[S];
  near_values<NB>(u, ny, nx, r, c, present, x);
  near_mad(x, present, n, mu, madu);
  near_values<NB>(v, ny, nx, r, c, present, x);
  near_mad(x, present, n, mv, madv);
  return true;
}

// substitute_alternatives! (src/quality.jl:307-351) at cell (r, c): judged
// against the snapshot outl_in; returns the new flag and may update u/v at
// the cell (it reads valid cells only, so in-place updates do not race).
// alt_u/alt_v hold nalt planes of G = ny*nx values. The medians of 1 and 2
// layers come from the register networks above, as in uod_cell: with indexed
// arrays in local memory a flagged cell's insertion sorts hold its warp: 3.0
// ms for the six sweeps of a sparsely seeded 4096 x 4096 series against 1.2.
// WIDE: 3 and 4 layers (er), whose arrays stay in local memory. Kernels take one
// form or the other: beside the networks' registers the wide one has a quarter of
// its warps (500 x 400 cells, 3 layers: 926 us in one kernel, 683 by itself).
template <bool WIDE>
__device__ __forceinline__ uint8_t substitute_cell(float* u, float* v, const uint8_t* outl_in, const uint8_t* gmask,
                                                   const float* alt_u, const float* alt_v, int nalt, int ny, int nx,
                                                   int r, int c, int er, double thr) {
  const int64_t G = (int64_t)ny * nx, k = r + (int64_t)c * ny;
  uint8_t o = outl_in[k];
  if (!o || (gmask && gmask[k])) return o;
  double mu, mv, madu, madv;
  if constexpr (!WIDE) {
    if (er == 1) {
      if (!near_spread<1>(u, v, ny, nx, r, c, outl_in, gmask, mu, mv, madu, madv)) return o;
    } else {
      if (!near_spread<2>(u, v, ny, nx, r, c, outl_in, gmask, mu, mv, madu, madv)) return o;
    }
  } else {
    double bu[UOD_MAXN], bv[UOD_MAXN], tu[UOD_MAXN], tv[UOD_MAXN];
    int n = 0;
    for (int c2 = max(0, c - er); c2 <= min(nx - 1, c + er); ++c2)
      for (int r2 = max(0, r - er); r2 <= min(ny - 1, r + er); ++r2) {
        if (r2 == r && c2 == c) continue;
        const int64_t q = r2 + (int64_t)c2 * ny;
        if (outl_in[q] || (gmask && gmask[q])) continue;
        bu[n] = (double)u[q];
        bv[n] = (double)v[q];
        ++n;
      }
    if (n < 3) return o;
    for (int i = 0; i < n; ++i) {
      tu[i] = bu[i];
      tv[i] = bv[i];
    }
    mu = median_d(tu, n);
    mv = median_d(tv, n);
    for (int i = 0; i < n; ++i) {
      tu[i] = fabs(__dsub_rn(bu[i], mu));
      tv[i] = fabs(__dsub_rn(bv[i], mv));
    }
    madu = median_d(tu, n);
    madv = median_d(tv, n);
  }
  for (int m = 0; m < nalt; ++m) {
    const float au = alt_u[k + m * G], av = alt_v[k + m * G];
    if (!(isfinite(au) && isfinite(av))) break;
    if (fabs(__dsub_rn((double)au, mu)) / __dadd_rn(madu, 0.1) <= thr &&
        fabs(__dsub_rn((double)av, mv)) / __dadd_rn(madv, 0.1) <= thr) {
      u[k] = au;
      v[k] = av;
      return 0;
    }
  }
  return o;
}

// replace_vectors! (src/quality.jl:85-114) support: growing square until >= 3
// valid neighbours, component-wise Float64 median.
constexpr int REPL_LOCAL = 64;

__device__ __forceinline__ bool repl_invalid(const uint8_t* flags, const uint8_t* gmask, int64_t q) {
  return (flags && flags[q]) || (gmask && gmask[q]);
}

// k-th smallest (0-based) of the valid values in a square, by counting;
// used only when a square holds more than REPL_LOCAL valid values.
static __device__ double select_square(const float* f, const uint8_t* flags, const uint8_t* gmask, int ny, int r0, int r1,
                                int c0, int c1, int kth) {
  for (int cc = c0; cc <= c1; ++cc)
    for (int rr = r0; rr <= r1; ++rr) {
      const int64_t q = rr + (int64_t)cc * ny;
      if (repl_invalid(flags, gmask, q)) continue;
      const double x = (double)f[q];
      int less = 0, le = 0;
      for (int c2 = c0; c2 <= c1; ++c2)
        for (int r2 = r0; r2 <= r1; ++r2) {
          const int64_t q2 = r2 + (int64_t)c2 * ny;
          if (repl_invalid(flags, gmask, q2)) continue;
          const double y = (double)f[q2];
          less += y < x;
          le += y <= x;
        }
      if (less <= kth && kth < le) return x;
    }
  return __longlong_as_double(0x7ff8000000000000LL);
}

static __device__ double median_square(const float* f, const uint8_t* flags, const uint8_t* gmask, int ny, int r0, int r1,
                                int c0, int c1, int n) {
  if (n <= REPL_LOCAL) {
    double buf[REPL_LOCAL];
    int m = 0;
    for (int cc = c0; cc <= c1; ++cc)
      for (int rr = r0; rr <= r1; ++rr) {
        const int64_t q = rr + (int64_t)cc * ny;
        if (repl_invalid(flags, gmask, q)) continue;
        buf[m++] = (double)f[q];
      }
    return median_d(buf, m);
  }
  for (int cc = c0; cc <= c1; ++cc)  // NaN anywhere -> NaN
    for (int rr = r0; rr <= r1; ++rr) {
      const int64_t q = rr + (int64_t)cc * ny;
      if (!repl_invalid(flags, gmask, q) && isnan(f[q])) return __longlong_as_double(0x7ff8000000000000LL);
    }
  if (n & 1) return select_square(f, flags, gmask, ny, r0, r1, c0, c1, n / 2);
  const double a = select_square(f, flags, gmask, ny, r0, r1, c0, c1, n / 2 - 1);
  const double b = select_square(f, flags, gmask, ny, r0, r1, c0, c1, n / 2);
  return __dadd_rn(a / 2.0, b / 2.0);
}


// Replacement of one invalid cell (invalid = flags | gmask); writes the new
// values through nu/nv (unchanged when no square holds 3 valid cells). The
// valid cells of a square are those of the one before and its ring, so a
// search that ends at radius r counts r^2 cells, not r^3.
__device__ __forceinline__ void replace_cell(const float* u, const float* v, const uint8_t* flags,
                                             const uint8_t* gmask, int ny, int nx, int r, int c, float& nu,
                                             float& nvv) {
  const int maxr = (ny > nx ? ny : nx) - 1;
  if (maxr < 1) return;
  const uint32_t present = near_present<1>(ny, nx, r, c, flags, gmask);
  int n = __popc(present);
  if (n >= 3) {  // nearly every cell: its 8 neighbours through the network
    float x[8];
    near_values<1>(u, ny, nx, r, c, present, x);
    nu = (float)median_net_d(x, n);
    near_values<1>(v, ny, nx, r, c, present, x);
    nvv = (float)median_net_d(x, n);
    return;
  }
  for (int rad = 2; rad <= maxr; ++rad) {
    const int r0 = max(0, r - rad), r1 = min(ny - 1, r + rad), c0 = max(0, c - rad), c1 = min(nx - 1, c + rad);
    for (int cc = c0; cc <= c1; ++cc) {
      if (cc == c - rad || cc == c + rad) {  // a column of the ring
        for (int rr = r0; rr <= r1; ++rr) n += !repl_invalid(flags, gmask, rr + (int64_t)cc * ny);
      } else {
        if (r - rad >= 0) n += !repl_invalid(flags, gmask, r - rad + (int64_t)cc * ny);
        if (r + rad < ny) n += !repl_invalid(flags, gmask, r + rad + (int64_t)cc * ny);
      }
    }
    if (n >= 3) {
      nu = (float)median_square(u, flags, gmask, ny, r0, r1, c0, c1, n);
      nvv = (float)median_square(v, flags, gmask, ny, r0, r1, c0, c1, n);
      return;
    }
  }
}

// smooth_field (src/quality.jl:123-136): separable [1 2 1]/4, replicated edges.
__device__ __forceinline__ float smooth_row(const float* f, int ny, int nx, int r, int c) {
  const float q = 0.25f;
  const int cl = c > 0 ? c - 1 : 0, cr = c < nx - 1 ? c + 1 : nx - 1;
  return FMUL(q, FADD(FADD(f[r + (int64_t)cl * ny], FMUL(2.0f, f[r + (int64_t)c * ny])), f[r + (int64_t)cr * ny]));
}
__device__ __forceinline__ float smooth_cell(const float* f, int ny, int nx, int r, int c) {
  const int rl = r > 0 ? r - 1 : 0, rr = r < ny - 1 ? r + 1 : ny - 1;
  const float tl = smooth_row(f, ny, nx, rl, c), t0 = smooth_row(f, ny, nx, r, c), tr = smooth_row(f, ny, nx, rr, c);
  return FMUL(0.25f, FADD(FADD(tl, FMUL(2.0f, t0)), tr));
}

// field_change key of one cell: max(|du|, |dv|) as its IEEE bits (all
// values are >= 0, so bits order like values), +Inf for a NaN transition,
// 0xFFFFFFFF (after every value) for cells that do not count.
__device__ __forceinline__ uint32_t change_key(float u, float v, float pu, float pv, bool masked, bool& counts) {
  counts = false;
  if (masked) return 0xFFFFFFFFu;
  const float du = fabsf(FSUB(u, pu)), dv = fabsf(FSUB(v, pv));
  if (isnan(du) || isnan(dv)) {
    if (isnan(u) == isnan(pu) && isnan(v) == isnan(pv)) return 0xFFFFFFFFu;
    counts = true;
    return 0x7F800000u;
  }
  counts = true;
  return __float_as_uint(fmaxf(du, dv));
}

// 95th percentile (Statistics.quantile! type 7) of n counted keys given the
// two order statistics it interpolates: index helper and final formula.
__device__ __forceinline__ void quantile95_index(int64_t n, int64_t& ka, int64_t& kb, double& g) {
  const double aleph = fma((double)n, 0.95, 0.05);
  int64_t j = (int64_t)trunc(aleph);
  const int64_t hi = n - 1 > 1 ? n - 1 : 1;
  j = j < 1 ? 1 : (j > hi ? hi : j);
  g = aleph - (double)j;
  g = g < 0 ? 0 : (g > 1 ? 1 : g);
  ka = n == 1 ? 0 : j - 1;
  kb = n == 1 ? 0 : j;
}
__device__ __forceinline__ float quantile95_value(uint32_t ka, uint32_t kb, double g) {
  const float a = __uint_as_float(ka), b = __uint_as_float(kb);
  double q;
  if (isfinite(a) && isfinite(b)) q = __dadd_rn((double)a, __dmul_rn(g, (double)FSUB(b, a)));
  else q = __dadd_rn(__dmul_rn(1.0 - g, (double)a), __dmul_rn(g, (double)b));
  return (float)q;
}

// 95th percentile of the counted keys of a grid by a 4 x 8-bit radix select,
// run by a cluster of FC_CLUSTER CTAs. key(i, counts) forms key i (change_key);
// the keys are kept in `keys` for the later digits. Each CTA counts the digits
// of its share in shared memory, a warp adding its equal digits at once (the
// leading digits of a converged field are nearly all equal), and every CTA adds
// up the cluster's counters, a thread per digit. The second order statistic
// is the first one or the least key above it. Latency bound: one CTA with a
// thread walking the 256 counters, twice, took 70 us at 127 x 127 cells against
// 14, and 1.4 ms for two of 1021 x 1021 against 0.41.
constexpr int FC_CLUSTER = 8, FC_THREADS = 512;

struct FieldChangeSmem {
  uint32_t hist[4][256];
  uint32_t digit, above, least, rank;
  uint32_t count[FC_THREADS / 32];
  uint32_t counted;
};

template <class Key>
__device__ __forceinline__ float cluster_field_change(FieldChangeSmem& sm, int64_t G, uint32_t* keys, const Key& key) {
  namespace cg = cooperative_groups;
  auto cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t i0 = (int64_t)cl.block_rank() * FC_THREADS + tid, step = (int64_t)FC_CLUSTER * FC_THREADS;
  for (int b = tid; b < 4 * 256; b += FC_THREADS) (&sm.hist[0][0])[b] = 0;
  if (tid == 0) {
    sm.counted = 0;
    sm.least = 0xFFFFFFFFu;
  }
  __syncthreads();
  // whole warps run every round: lanes past the end take part in the matches
  const int64_t rounds = (G + step - 1) / step;
  uint32_t prefix = 0, pmask = 0;
  int64_t n = 0, k = 0, kb = 0;
  double g = 0;
  for (int d = 0; d < 4; ++d) {
    const int shift = 24 - 8 * d;
    uint32_t here = 0;
    int64_t i = i0;
    for (int64_t q = 0; q < rounds; ++q, i += step) {
      uint32_t x = 0;
      bool in = i < G;
      if (d == 0) {
        bool counts = false;
        if (in) keys[i] = x = key(i, counts);
        here += counts;
      } else if (in) {
        x = keys[i];
      }
      in = in && (x & pmask) == prefix;
      const uint32_t digit = in ? (x >> shift) & 255u : 256u;
      const uint32_t same = __match_any_sync(0xFFFFFFFFu, digit);
      if (in && (same & ((1u << lane) - 1u)) == 0) atomicAdd(&sm.hist[d][digit], (uint32_t)__popc(same));
    }
    if (d == 0) {
      here = __reduce_add_sync(0xFFFFFFFFu, here);
      if (lane == 0 && here) atomicAdd(&sm.counted, here);
    }
    cl.sync();
    if (d == 0) {
      for (int q = 0; q < FC_CLUSTER; ++q) n += cl.map_shared_rank(&sm, q)->counted;
      if (n == 0) break;  // the same in every CTA
      quantile95_index(n, k, kb, g);
      kb -= k;  // 0 or 1
    }
    uint32_t cnt = 0, upto = 0;
    if (tid < 256) {
      for (int q = 0; q < FC_CLUSTER; ++q) cnt += cl.map_shared_rank(&sm, q)->hist[d][tid];
      upto = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, upto, o);
        if (lane >= o) upto += t;
      }
      if (lane == 31) sm.count[warp] = upto;
    }
    __syncthreads();
    if (tid < 256) {
      for (int w = 0; w < warp; ++w) upto += sm.count[w];
      const uint32_t before = upto - cnt;
      if ((int64_t)before <= k && k < (int64_t)upto) {
        sm.digit = (uint32_t)tid;
        sm.rank = (uint32_t)(k - before);
        sm.above = cnt;
      }
    }
    __syncthreads();
    prefix |= sm.digit << shift;
    pmask |= 255u << shift;
    k = sm.rank;
  }
  float change = 0.f;
  if (n > 0) {
    uint32_t b = prefix;
    if (kb && k + 1 >= (int64_t)sm.above) {  // the same in every CTA
      uint32_t least = 0xFFFFFFFFu;
      for (int64_t i = i0; i < G; i += step) {
        const uint32_t x = keys[i];
        if (x > prefix) least = min(least, x);
      }
      least = __reduce_min_sync(0xFFFFFFFFu, least);
      if (lane == 0) atomicMin(&sm.least, least);
      cl.sync();
      for (int q = 0; q < FC_CLUSTER; ++q) least = min(least, cl.map_shared_rank(&sm, q)->least);
      b = least;
    }
    change = quantile95_value(prefix, b, g);
  }
  cl.sync();  // no CTA leaves while its counters are read
  return change;
}

}  // namespace hh
