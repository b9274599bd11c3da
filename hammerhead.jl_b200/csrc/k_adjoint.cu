// Adjoint of deformation + zero-lag correlation (sm_100a).
//
// Loss of a predictor field P = (u, v) on a uniform node grid:
//   L(P) = - sum over windows j of NCC0_j,
//   NCC0_j = sum (a - abar)(b - bbar) / sqrt(sum (a - abar)^2 sum (b - bbar)^2)
// over the W x W pixels of window j of the pair deformed by P exactly as a
// WIDIM sweep deforms it (bilinear predictor with flat extrapolation, cubic
// B-spline samples at -+ (u, v)/2; deform_columns!, src/pipeline.jl:957-965).
//
// Three launches (and the loss), no atomics, no stored deformed image:
//   1. per tile of neighbouring windows (one CTA): the tile's pixels deformed
//      once into shared memory, then FP64 moments and the window constants of
//      the gradient, a warp per window;
//   2. per pixel: recompute the deformed samples and their B-spline
//      derivatives, sum dL/da, dL/db over the windows holding the pixel,
//      chain through -+ 1/2 to the pixel displacement gradient (gu, gv);
//   3. per node: the transpose of the bilinear predictor interpolation,
//      gathered over the node's support in FP64, axis by axis.
// Bound by issue. Windows at 50 % overlap share each pixel four times; a CTA
// per window deformed it each time and spent as long on its ten block-wide
// barriers. The predictor's cell and fraction along an axis (two divisions)
// depend on the row or the column alone, so they are formed once per row and
// column of a tile, and the B-spline weights divide by 6 without a division.
// 1024^2, 16 px windows at 50 %, P 127 x 127, loss and gradient: 295 us a
// call in the earlier form, 113 us now.
#include <math.h>
#include <stdint.h>

#include "hh_internal.h"
#include "hh_spline.cuh"

namespace hh {

namespace {

__device__ __forceinline__ void cubw_f(float d, float* w) {
  const float x3 = d * d * d, c = 1.f - d, c3 = c * c * c;
  w[0] = div6(c3);
  w[1] = 2.f / 3.f - d * d + x3 / 2.f;
  w[2] = 2.f / 3.f - c * c + c3 / 2.f;
  w[3] = div6(x3);
}
// d/dd of the cubic B-spline weights
__device__ __forceinline__ void cubw_df(float d, float* w) {
  const float c = 1.f - d;
  w[0] = -0.5f * c * c;
  w[1] = -2.f * d + 1.5f * d * d;
  w[2] = 2.f * c - 1.5f * c * c;
  w[3] = 0.5f * d * d;
}

// zero-extrapolated cubic B-spline sample at 1-based (yy, xx); with GRAD
// also its derivatives along rows (gy) and columns (gx)
template <bool GRAD>
__device__ __forceinline__ float bs_sample(const float* __restrict__ C, int64_t nr, int64_t nc, float yy, float xx,
                                           float& gy, float& gx) {
  gy = gx = 0.f;
  if (yy < 1.f || yy > (float)nr || xx < 1.f || xx > (float)nc) return 0.f;
  // a NaN coordinate (from the predictor) takes the first cell; its weights make the sample NaN
  const int64_t iy = min((int64_t)fmaxf(floorf(yy), 1.f), nr - 1);
  const int64_t ix = min((int64_t)fmaxf(floorf(xx), 1.f), nc - 1);
  float wy[4], wx[4], dy[4], dx[4];
  cubw_f(yy - (float)iy, wy);
  cubw_f(xx - (float)ix, wx);
  if (GRAD) {
    cubw_df(yy - (float)iy, dy);
    cubw_df(xx - (float)ix, dx);
  }
  const int64_t ld = nr + 2;
  const float* base = C + (iy - 1) + (ix - 1) * ld;
  float s = 0.f, sy = 0.f, sx = 0.f;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    float t = 0.f, tx = 0.f;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float c = __ldg(base + a + b * ld);
      t += wx[b] * c;
      if (GRAD) tx += dx[b] * c;
    }
    s += wy[a] * t;
    if (GRAD) {
      sy += dy[a] * t;
      sx += wy[a] * tx;
    }
  }
  gy = sy;
  gx = sx;
  return s;
}

// Gridded(Linear()) + Flat() along one axis (as the deformation kernel)
__device__ __forceinline__ void lin_axis_f(float q, float q0, float step, int n, int& i, float& d) {
  if (n == 1) { i = 0; d = 0.f; return; }
  const float last = __fadd_rn(q0, __fmul_rn((float)(n - 1), step));
  if (q <= q0) { i = 0; d = 0.f; return; }
  if (q >= last) { i = n - 2; d = 1.f; return; }
  i = (int)floorf(__fdiv_rn(__fsub_rn(q, q0), step));
  if (i > n - 2) i = n - 2;
  const float k0 = __fadd_rn(q0, __fmul_rn((float)i, step)), k1 = __fadd_rn(q0, __fmul_rn((float)(i + 1), step));
  d = __fdiv_rn(__fsub_rn(q, k0), __fsub_rn(k1, k0));
}

// where a pixel row or column falls on the predictor's nodes
struct Cell {
  int i;    // cell
  float d;  // fraction
};
__device__ __forceinline__ Cell cell_at(float q, float q0, float step, int n) {
  Cell c;
  lin_axis_f(q, q0, step, n, c.i, c.d);
  return c;
}

__device__ __forceinline__ float bilin(const float* f, const NccArgs& a, Cell y, Cell x) {
  const int iy2 = a.gny == 1 ? y.i : y.i + 1, ix2 = a.gnx == 1 ? x.i : x.i + 1;
  const float f00 = f[y.i + x.i * a.gny], f01 = f[y.i + ix2 * a.gny], f10 = f[iy2 + x.i * a.gny],
              f11 = f[iy2 + ix2 * a.gny];
  const float p = __fadd_rn(__fmul_rn(__fsub_rn(1.f, x.d), f00), __fmul_rn(x.d, f01));
  const float q = __fadd_rn(__fmul_rn(__fsub_rn(1.f, x.d), f10), __fmul_rn(x.d, f11));
  return __fadd_rn(__fmul_rn(__fsub_rn(1.f, y.d), p), __fmul_rn(y.d, q));
}

// deformed samples of pixel (r, c) (0-based) of both frames
template <bool GRAD>
__device__ __forceinline__ void deformed(const NccArgs& a, int64_t r, int64_t c, Cell y, Cell x, float& va, float& vb,
                                         float& ay, float& ax, float& by, float& bx) {
  const float R = (float)(r + 1), Cc = (float)(c + 1);
  const float u2 = __fmul_rn(bilin(a.P, a, y, x), 0.5f);
  const float v2 = __fmul_rn(bilin(a.P + (int64_t)a.gny * a.gnx, a, y, x), 0.5f);
  va = bs_sample<GRAD>(a.CA, a.nr, a.nc, __fsub_rn(R, v2), __fsub_rn(Cc, u2), ay, ax);
  vb = bs_sample<GRAD>(a.CB, a.nr, a.nc, __fadd_rn(R, v2), __fadd_rn(Cc, u2), by, bx);
}

// The CTA's place in a two-dimensional arrangement of nx (first axis, fastest)
// by as many as there are. The launches are one-dimensional: a grid's second
// dimension ends at 65535, which image columns and node columns may pass.
struct Block {
  int x, y;
};
__device__ __forceinline__ Block block_of(int64_t nx) {
  const int n = (int)nx;
  return Block{(int)blockIdx.x % n, (int)blockIdx.x / n};
}

constexpr int NCC_THREADS = 256;

__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < NCC_THREADS / 32; ++w) t += red[w];
  return t;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Windows of a tile along one axis: as many as fit the side, but at least
// NCC_TILES tiles where the image has them. 64 px (a tile's deformed pixels,
// float2, take 33 KB) leave 6 CTAs per SM and, at 1024^2 with 16 px windows,
// more CTAs than SMs, while a pixel is deformed 1.3 times on average; sides of
// 96 px deform 1.2 times but leave one CTA per SM there (53 us against 40 us).
// Windows above 32 px need the larger side to share. On small images the
// longest tiles leave a few CTAs with all the windows: loss alone with 13 px
// windows at every pixel of 92 x 61, 2 tiles 465 us, 260 tiles 32, 3920 (a
// window each) 59; 16 px at 50 % of 256^2, 25 tiles 45 us, 256 tiles 33; 512^2,
// 81 tiles 44, 256 tiles 34. Above some 250 tiles the sides decide.
constexpr int NCC_SIDE = 96;  // the longest
constexpr int64_t NCC_TILES = 256;
static int64_t tiles_of(const NccArgs& a, int TW) {
  return (int64_t)((a.wy + TW - 1) / TW) * ((a.wx + TW - 1) / TW);
}
static int tile_windows(const NccArgs& a) {
  int TW = 1 + ((a.W <= 32 ? 64 : NCC_SIDE) - a.W) / a.step;
  while (TW > 1 && tiles_of(a, TW) < NCC_TILES) --TW;
  return TW;
}
__host__ __device__ __forceinline__ int tile_side(int W, int step, int TW) { return W + (TW - 1) * step; }
static size_t tile_smem(int W, int step, int TW) {
  const size_t n = tile_side(W, step, TW);
  return n * (n + 1) * sizeof(float2) + 2 * n * sizeof(Cell) + NCC_THREADS / 32 * sizeof(double);
}

// 1. window constants: ncc, abar, bbar, inv = 1/sqrt(Saa Sbb), ca = ncc/Saa, cb = ncc/Sbb;
//    and per CTA the sum of its ncc (after the constants of all windows)
__global__ void __launch_bounds__(NCC_THREADS) ncc_tile_kernel(const NccArgs a, int TW) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int W = a.W, n = W * W, side = tile_side(W, a.step, TW), ld = side + 1;
  float2* T = reinterpret_cast<float2*>(smem_raw);  // column c of the tile at c * ld
  Cell* ry = reinterpret_cast<Cell*>(T + side * ld);
  Cell* cx = ry + side;
  double* part = reinterpret_cast<double*>(cx + side);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Block b = block_of((a.wy + TW - 1) / TW);
  const int jr0 = b.x * TW, jc0 = b.y * TW;
  const int ty = min(TW, a.wy - jr0), tx = min(TW, a.wx - jc0);           // windows of this tile
  const int rt = W + (ty - 1) * a.step, ct = W + (tx - 1) * a.step;       // its pixels
  const int64_t r0 = (int64_t)jr0 * a.step, c0 = (int64_t)jc0 * a.step;
  for (int k = tid; k < rt + ct; k += NCC_THREADS) {
    if (k < rt) ry[k] = cell_at((float)(r0 + k + 1), a.y0, a.ysp, a.gny);
    else cx[k - rt] = cell_at((float)(c0 + k - rt + 1), a.x0, a.xsp, a.gnx);
  }
  __syncthreads();
  // k / rt as a multiplication, exact for k rt < 2^22 (k < 96^2)
  const uint32_t inv_rt = (1u << 22) / rt + 1;
  for (int k = tid; k < rt * ct; k += NCC_THREADS) {
    const int c = (int)(((uint32_t)k * inv_rt) >> 22), r = k - c * rt;
    float2 v;
    float d0, d1, d2, d3;
    deformed<false>(a, r0 + r, c0 + c, ry[r], cx[c], v.x, v.y, d0, d1, d2, d3);
    T[c * ld + r] = v;
  }
  __syncthreads();
  const uint32_t inv_w = (1u << 20) / W + 1;  // k / W, exact for k W < 2^20 (k < 64^2)
  double loss = 0.0;
  for (int w = warp; w < ty * tx; w += NCC_THREADS / 32) {
    const int wr = w % ty, wc = w / ty;
    const float2* B = T + wc * a.step * ld + wr * a.step;
    double sa = 0.0, sb = 0.0;
#pragma unroll 4
    for (int k = lane; k < n; k += 32) {
      const int q = (int)(((uint32_t)k * inv_w) >> 20);
      const float2 v = B[q * ld + k - q * W];
      sa += (double)v.x;
      sb += (double)v.y;
    }
    const double ma = warp_sum_d(sa) / n, mb = warp_sum_d(sb) / n;
    double saa = 0.0, sbb = 0.0, sab = 0.0;
#pragma unroll 4
    for (int k = lane; k < n; k += 32) {
      const int q = (int)(((uint32_t)k * inv_w) >> 20);
      const float2 v = B[q * ld + k - q * W];
      const double da = (double)v.x - ma, db = (double)v.y - mb;
      saa += da * da;
      sbb += db * db;
      sab += da * db;
    }
    saa = warp_sum_d(saa);
    sbb = warp_sum_d(sbb);
    sab = warp_sum_d(sab);
    const bool flat = !(saa > 0 && sbb > 0);  // a flat window contributes nothing
    const double inv = flat ? 0.0 : 1.0 / sqrt(saa * sbb), ncc = flat ? 0.0 : sab * inv;
    loss += ncc;
    if (lane == 0) {
      double* o = a.wstat + 6 * ((int64_t)(jr0 + wr) + (int64_t)(jc0 + wc) * a.wy);
      o[0] = ncc;
      o[1] = flat ? 0.0 : ma;
      o[2] = flat ? 0.0 : mb;
      o[3] = inv;
      o[4] = flat ? 0.0 : ncc / saa;
      o[5] = flat ? 0.0 : ncc / sbb;
    }
  }
  if (lane == 0) part[warp] = loss;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int k = 0; k < NCC_THREADS / 32; ++k) t += part[k];
    a.wstat[6 * (int64_t)a.wy * a.wx + blockIdx.x] = t;
  }
}

// 2. pixel displacement gradient (gu, gv) = dL/d(u, v) at every pixel: a
//    thread keeps its row and walks PC columns, so what belongs to a row
//    (predictor cell, windows that hold it) or to a column is formed once.
//    PC = 8 columns where that leaves NCC_PBLOCKS CTAs, fewer on small images,
//    whose threads would be too few: loss and gradient with 49 px windows at
//    every pixel of 86 x 76, 8 columns (10 CTAs) 393 us, one 110; 16 px windows
//    at every pixel of 76 x 71 181 and 65 us; 16 px at 50 % of 256^2 52 and 51.
constexpr int NCC_PR = 128, NCC_PC = 8;  // NCC_PC: the most columns of a thread
constexpr int64_t NCC_PBLOCKS = 296;
struct Span {
  int j0, j1;  // windows j0..j1 hold the row or column
};
__device__ __forceinline__ Span span_at(int64_t p, int W, int step, int nw) {
  return Span{p < W ? 0 : (int)((p - W) / step + 1), min(nw - 1, (int)(p / step))};
}
__global__ void __launch_bounds__(NCC_PR) ncc_pixel_kernel(const NccArgs a, int PC) {
  __shared__ Cell cx[NCC_PC];
  __shared__ Span cw[NCC_PC];
  const Block b = block_of((a.nr + NCC_PR - 1) / NCC_PR);
  const int64_t P = a.nr * a.nc, r = (int64_t)b.x * NCC_PR + threadIdx.x, c0 = (int64_t)b.y * PC;
  const int nc = (int)min((int64_t)PC, a.nc - c0);
  if (threadIdx.x < nc) {
    cx[threadIdx.x] = cell_at((float)(c0 + threadIdx.x + 1), a.x0, a.xsp, a.gnx);
    cw[threadIdx.x] = span_at(c0 + threadIdx.x, a.W, a.step, a.wx);
  }
  __syncthreads();
  // the rows' and columns' cells, for the node kernel (the columns' also where
  // the image has fewer rows than the block has columns)
  if (b.x == 0 && threadIdx.x < nc) {
    a.cells[2 * (a.nr + c0 + threadIdx.x)] = cx[threadIdx.x].i;
    a.cells[2 * (a.nr + c0 + threadIdx.x) + 1] = __float_as_int(cx[threadIdx.x].d);
  }
  if (r >= a.nr) return;
  const Cell y = cell_at((float)(r + 1), a.y0, a.ysp, a.gny);
  if (b.y == 0) {
    a.cells[2 * r] = y.i;
    a.cells[2 * r + 1] = __float_as_int(y.d);
  }
  const Span rw = span_at(r, a.W, a.step, a.wy);
  // dL/da = sum_j -(b - bbar_j) inv_j + ca_j (a - abar_j) over the windows j
  // that hold the pixel, dL/db likewise: the sums of the constants change only
  // with the set of windows, every `step` columns
  double si = 0.0, sca = 0.0, scb = 0.0, ka = 0.0, kb = 0.0;
  for (int k = 0; k < nc; ++k) {
    const int64_t c = c0 + k;
    if (k == 0 || cw[k].j0 != cw[k - 1].j0 || cw[k].j1 != cw[k - 1].j1) {
      si = sca = scb = ka = kb = 0.0;
      for (int jc = cw[k].j0; jc <= cw[k].j1; ++jc)
        for (int jr = rw.j0; jr <= rw.j1; ++jr) {
          const double* s = a.wstat + 6 * ((int64_t)jr + (int64_t)jc * a.wy);
          si += s[3];
          sca += s[4];
          scb += s[5];
          ka += s[2] * s[3] - s[4] * s[1];
          kb += s[1] * s[3] - s[5] * s[2];
        }
    }
    float gu = 0.f, gv = 0.f;
    if (rw.j0 <= rw.j1 && cw[k].j0 <= cw[k].j1) {
      float va, vb, ay, ax, by, bx;
      deformed<true>(a, r, c, y, cx[k], va, vb, ay, ax, by, bx);
      const double ga = sca * (double)va - si * (double)vb + ka, gb = scb * (double)vb - si * (double)va + kb;
      const float fa = (float)ga, fb = (float)gb;
      gu = fa * (-0.5f * ax) + fb * (0.5f * bx);
      gv = fa * (-0.5f * ay) + fb * (0.5f * by);
    }
    a.gpix[r + c * a.nr] = gu;
    a.gpix[P + r + c * a.nr] = gv;
  }
}

// 3. dL/dP at every node: the transpose of the bilinear interpolation, axis by
//    axis. A CTA takes NODE_R x NODE_C nodes and walks the image columns of
//    their support NODE_K at a time: first each (node row, column) sums its
//    rows, then each node its columns. (A warp per node read every pixel of a
//    node's support for itself, a third of its lanes idle, and formed the
//    weights again for each node: 48 us at 1024^2 against 21 us.)
constexpr int NODE_R = 16, NODE_C = 2, NODE_K = 32, NODE_THREADS = 256;
struct Reach {
  int64_t lo, hi;  // 1-based pixels whose stencil may reach the node
};
__device__ __forceinline__ Reach reach_of(int g, int n, float q0, float step, int64_t np) {
  return Reach{g == 0 ? 1 : max((int64_t)1, (int64_t)floorf(q0 + (g - 1) * step)),
               g == n - 1 ? np : min(np, (int64_t)ceilf(q0 + (g + 1) * step))};
}
// weight of node g in the cell of pixel p (0-based), which has n nodes
__device__ __forceinline__ float cell_w(const int* cells, int64_t p, int g, int n) {
  const int i = cells[2 * p];
  const float d = __int_as_float(cells[2 * p + 1]);
  return (i == g ? 1.f - d : 0.f) + ((n == 1 ? i : i + 1) == g ? d : 0.f);
}
__global__ void __launch_bounds__(NODE_THREADS) ncc_node_kernel(const NccArgs a) {
  __shared__ double t[2][NODE_K][NODE_R + 1];
  const int64_t G = (int64_t)a.gny * a.gnx, P = a.nr * a.nc;
  const Block b = block_of((a.gny + NODE_R - 1) / NODE_R);
  const int gy0 = b.x * NODE_R, gx0 = b.y * NODE_C;
  const int64_t c_lo = reach_of(gx0, a.gnx, a.x0, a.xsp, a.nc).lo;
  const int64_t c_hi = reach_of(min(gx0 + NODE_C, a.gnx) - 1, a.gnx, a.x0, a.xsp, a.nc).hi;
  // this thread's node and component in the second step
  const int ny = threadIdx.x % NODE_R, nx = threadIdx.x / NODE_R % NODE_C, comp = threadIdx.x / (NODE_R * NODE_C);
  const int gx = gx0 + nx;
  const bool node = comp < 2 && gy0 + ny < a.gny && gx < a.gnx;
  const Reach cr = reach_of(min(gx, a.gnx - 1), a.gnx, a.x0, a.xsp, a.nc);
  double acc = 0.0;
  for (int64_t cb = c_lo; cb <= c_hi; cb += NODE_K) {
    for (int e = threadIdx.x; e < NODE_R * NODE_K; e += NODE_THREADS) {
      const int gy = gy0 + e % NODE_R, k = e / NODE_R;
      double su = 0.0, sv = 0.0;
      if (gy < a.gny && cb + k <= c_hi) {
        const Reach rr = reach_of(gy, a.gny, a.y0, a.ysp, a.nr);
        const float* g = a.gpix + (cb + k - 1) * a.nr - 1;
#pragma unroll 6
        for (int64_t R = rr.lo; R <= rr.hi; ++R) {
          const float w = cell_w(a.cells, R - 1, gy, a.gny);
          const bool on = w != 0.f;  // a pixel without weight does not count (it may hold NaN)
          su += (double)w * (double)(on ? g[R] : 0.f);
          sv += (double)w * (double)(on ? g[P + R] : 0.f);
        }
      }
      t[0][k][e % NODE_R] = su;
      t[1][k][e % NODE_R] = sv;
    }
    __syncthreads();
    const int k0 = (int)max((int64_t)0, cr.lo - cb), k1 = (int)min((int64_t)NODE_K - 1, cr.hi - cb);
    for (int k = k0; node && k <= k1; ++k) {
      const float w = cell_w(a.cells, a.nr + cb + k - 1, gx, a.gnx);
      if (w != 0.f) acc += (double)w * t[comp][k][ny];
    }
    __syncthreads();
  }
  if (node) a.grad[comp * G + (gy0 + ny) + (int64_t)gx * a.gny] = (float)acc;
}

// loss = -sum of the tiles' sums (one CTA)
__global__ void __launch_bounds__(NCC_THREADS) ncc_loss_kernel(const NccArgs a, int64_t ntiles) {
  __shared__ double red[NCC_THREADS / 32];
  const double* part = a.wstat + 6 * (int64_t)a.wy * a.wx;
  double s = 0.0;
  for (int64_t j = threadIdx.x; j < ntiles; j += NCC_THREADS) s += part[j];
  s = block_sum(s, red);
  if (threadIdx.x == 0) *a.loss = -s;
}

}  // namespace

int64_t ncc_wstat_words(int32_t wy, int32_t wx) { return 7 * (int64_t)wy * wx; }  // at most a tile per window

cudaError_t launch_ncc_loss_grad(const NccArgs& a, cudaStream_t s) {
  if (a.wy < 1 || a.wx < 1 || a.W < 2 || a.W > 64 || a.step < 1) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(ncc_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(NCC_SIDE * (NCC_SIDE + 1) * sizeof(float2) + 4096));
  if (e != cudaSuccess) return e;
  auto blocks = [](int64_t n, int per) { return (n + per - 1) / per; };
  const int TW = tile_windows(a);
  const int64_t tiles = tiles_of(a, TW);
  int PC = NCC_PC;
  while (PC > 1 && blocks(a.nr, NCC_PR) * blocks(a.nc, PC) < NCC_PBLOCKS) PC /= 2;
  const int64_t px = blocks(a.nr, NCC_PR) * blocks(a.nc, PC), nodes = blocks(a.gny, NODE_R) * blocks(a.gnx, NODE_C);
  if (tiles > INT32_MAX || (a.grad && (px > INT32_MAX || nodes > INT32_MAX))) return cudaErrorInvalidValue;
  ncc_tile_kernel<<<(unsigned)tiles, NCC_THREADS, tile_smem(a.W, a.step, TW), s>>>(a, TW);
  ncc_loss_kernel<<<1, NCC_THREADS, 0, s>>>(a, tiles);
  if (a.grad) {
    ncc_pixel_kernel<<<(unsigned)px, NCC_PR, 0, s>>>(a, PC);
    ncc_node_kernel<<<(unsigned)nodes, NODE_THREADS, 0, s>>>(a);
  }
  return cudaGetLastError();
}

}  // namespace hh
