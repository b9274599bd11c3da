// Symmetric image deformation for WIDIM sweeps (sm_100a).
//
// prefilter: cubic B-spline coefficients of Interpolations.jl's
//   BSpline(Cubic(Line(OnGrid()))) on the (nr+2) x (nc+2) padded index set
//   (the coefficient array image_interpolant builds, src/pipeline.jl:75-85,
//   909-915): per line, rows [1 4 1]/6 inside and the "Line" boundary rows
//   c0 - 2c1 + c2 = 0. Eliminating the boundary rows leaves c1 = b1,
//   c_{n-2} = b_{n-2} and a constant-coefficient tridiagonal system, solved
//   by the Thomas algorithm with the line-independent elimination factors
//   precomputed once. Separable: every column, then every row.
// deform: a lane per image row, stepping along the columns, evaluates the
//   predictor by bilinear interpolation with flat extrapolation (Gridded(Linear()) + Flat(),
//   src/pipeline.jl:561-600) and samples both coefficient arrays with the
//   4x4 cubic B-spline at -+ half the displacement, zero outside the image
//   (deform_columns!, src/pipeline.jl:957-965; _ka_deform!,
//   src/ka_backend.jl:266-312).
// All floating-point operations use explicit round-to-nearest intrinsics so
// no multiply-add is fused: results equal the CPU restatement bit for bit.
#include <math.h>
#include <stdint.h>

#include "hh_attr.h"
#include "hh_batch.h"
#include "hh_internal.h"
#include "hh_pred.cuh"
#include "hh_spline.cuh"

namespace hh {

// Correctly rounded float constants of 1/6 and 2/3 (what 1f0/6 and 2f0/3
// evaluate to), and x/2 taken as x*0.5: halving by a power of two is the
// same correctly rounded value either way, so the results are unchanged.
static __device__ __forceinline__ float k_sixth() { return __int_as_float(0x3E2AAAAB); }
static __device__ __forceinline__ float k_two_thirds() { return __int_as_float(0x3F2AAAAB); }
#define kSixth k_sixth()
#define kTwoThirds k_two_thirds()

// Elimination factors for a line of padded length n: unknown rows
// i = 3..n-2 (1-based). inv[k] = 1/den_k, cp[k] = (1/6)*inv[k], k = i - 3.
__global__ void bspline_factors_kernel(int64_t n, float* cp, float* inv) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const float sixth = FD(1.0f, 6.0f), b = FD(4.0f, 6.0f);
  const int64_t m = n - 4;  // number of unknowns
  float cprev = 0.f;
  for (int64_t k = 0; k < m; ++k) {
    float den = k == 0 ? b : FS(b, FM(sixth, cprev));
    float iv = FD(1.0f, den);
    inv[k] = iv;
    cprev = FM(sixth, iv);
    cp[k] = cprev;
  }
}

// Both Thomas sweeps are contractions (|cp_k| -> 0.268), so each line is cut
// into independent segments of BS_SEG unknowns whose sweeps start BS_WARM
// unknowns early from a zero state; the neglected term is below
// 0.268^32 ~ 5e-19 of the value, far under float rounding. The CPU
// restatement solves each line in one sweep; the deformed images are held to
// 4 ulp of the image scale against it. The forward sweep is
// d_k = (rhs_k - d_{k-1}/6) inv_k (unknown k at line element k + 2; rhs_0 and
// rhs_{m-1} carry the known c1 and c_{n-2}), the backward sweep
// x_k = d_k - cp_k x_{k+1}, followed by the "Line" boundary coefficients
// c0 = 2c1 - c2 and c_{n-1} = 2c_{n-2} - c_{n-3}. BS_SEG, BS_WARM and the
// segment count b_nseg are in hh_internal.h (the batched plan counts work
// items with them).

cudaError_t launch_bspline_factors(int64_t n, float* cp, float* inv, cudaStream_t s) {
  bspline_factors_kernel<<<1, 1, 0, s>>>(n, cp, inv);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Two floats in one register pair: the frames' samples A and B, or the
// predictor's components u and v, go through the same arithmetic, and the
// packed instructions issue it once for both. Each half is rounded to nearest
// like the scalar operation.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pk(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpk(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 both(float x) { return pk(x, x); }
// Packed products, each rounded by itself: the assembler contracts a packed
// multiplication and the addition that uses it into one rounding, so a product
// is the fused operation with an addend of -0 that only the launch knows.
struct Mul2 {
  F2 zero;
  __device__ __forceinline__ F2 operator()(F2 a, F2 b) const { return fma2(a, b, zero); }
};
// div6 of both halves (its remainder step as q0 * -6 + x, the same product)
__device__ __forceinline__ F2 div6_2(const Mul2& mul2, F2 x) {
  const F2 r = both(k_sixth()), q0 = mul2(x, r);
  return fma2(fma2(q0, both(-6.0f), x), r, q0);
}
// Interpolations' cubic B-spline weights at fractional offsets d.
__device__ __forceinline__ void cubw2(const Mul2& mul2, F2 d, F2* w) {
  const F2 d2 = mul2(d, d), x3 = mul2(d2, d), c = sub2(both(1.f), d), c2 = mul2(c, c), c3 = mul2(c2, c);
  const F2 two3 = both(kTwoThirds), half = both(0.5f);
  w[0] = div6_2(mul2, c3);
  w[1] = add2(sub2(two3, d2), mul2(x3, half));
  w[2] = add2(sub2(two3, c2), mul2(c3, half));
  w[3] = div6_2(mul2, x3);
}

// where coordinate q of a sample starts on an axis of n pixels: the cell's
// first coefficient, and whether the sample is inside the image. A sample
// outside reads the nearest cell and counts as zero.
__device__ __forceinline__ int spline_cell(float q, int n, bool& in) {
  in = !(q < 1.f || q > (float)n);
  return min(__float2int_rd(fminf(fmaxf(q, 1.f), (float)n)), n - 1);
}

// One warp deforms both frames on a strip of 32 rows and `cols` columns: a lane
// per row, stepping along the columns, so that every load and store of the warp
// runs down one column. The predictor's cell and fraction are formed once per row
// and, a lane each, once per column; its corner values are loaded where the
// columns enter a new cell.
// WRAP, for images whose last strip of rows would leave more than a fifth of the
// lanes idle: a lane takes a row slot, the rows of one block of `cols` columns
// followed by those of the next. A warp then has two blocks where it passes from
// one to the next, or several if the image has fewer than 32 rows.
//
// What bounds it: the latency of a column's chain (coordinates, 32 loads, the
// sums) at 24 warps per SM, then instructions issued (61 % of the slots): a
// pixel needs two samples of 16 coefficients, whose products and sums may not
// be fused (they are the CPU restatement's), and four cubic weights, some 270
// instructions in packed form. 2048 x 2048: a thread per pixel with its own
// divisions and 64-bit indices took 79 us; four rows per thread, whose loads
// touch four lines each, 70; this takes 52. Strips of 8 columns: 16 and 32 are
// as fast there (51, 59 us); 64 registers for 32 warps per SM spill and gain
// nothing (51 us). Images with fewer than DEF_STRIPS strips take fewer columns,
// since a strip's columns are one chain: 100 x 100 12.5 us with 8 columns, 6.9
// with one; 512 x 512 10.8, 9.7 with 4; 768 x 1024 16.6, 19.0 with 4 (a pixel's
// share of the cells grows). WRAP: 12 x 36000 20.6 -> 17.0 us, 33 x 33000 30.8 ->
// 26.9; 2048 x 2048 would take 54.3 instead of 52.2.
constexpr int DEF_COLS = 8;  // the most columns of a strip
constexpr int64_t DEF_STRIPS = 148 * 10;
__host__ __device__ static inline int64_t def_row_strips(int64_t nr) { return (nr + 31) / 32; }
// columns per strip of an image of nr rows where the launch asks for cols: with
// WRAP a strip's columns fit the lanes that form their cells (at most 31 / nr + 2
// blocks)
__host__ __device__ static inline int def_cols(bool wrap, int64_t nr, int cols) {
  while (wrap && cols > 1 && (31 / nr + 2) * cols > 32) cols /= 2;
  return cols;
}
__host__ __device__ static inline int64_t def_strips(bool wrap, int64_t nr, int64_t nc, int cols) {
  const int n = def_cols(wrap, nr, cols);
  const int64_t blocks = (nc + n - 1) / n;
  return wrap ? (nr * blocks + 31) / 32 : def_row_strips(nr) * blocks;
}
template <bool WRAP>
__device__ __forceinline__ void deform_strip(const float* __restrict__ CA, const float* __restrict__ CB, int nr, int nc,
                                             const float* __restrict__ pu, const float* __restrict__ pv,
                                             const PredGrid& g, float* __restrict__ wA, float* __restrict__ wB,
                                             int64_t strip, int cols, float minus_zero) {
  const Mul2 mul2{both(minus_zero)};
  const int lane = threadIdx.x & 31;
  const int64_t ld = (int64_t)nr + 2;
  int r, c00, c0, c1;  // row; the strip's first column, and this lane's columns [c0, c1)
  bool store = true;
  if (WRAP) {
    const int b0 = (int)(strip * 32 / nr), v = (int)(strip * 32 - (int64_t)b0 * nr) + lane;
    r = v % nr;
    c00 = b0 * cols;
    c0 = c00 + v / nr * cols;
    c1 = c0 + cols;
  } else {
    const int64_t rs = def_row_strips(nr);
    const int rl = (int)(strip % rs) * 32 + lane;
    r = min(rl, nr - 1);
    store = rl < nr;
    c00 = c0 = (int)(strip / rs) * cols;
    c1 = min(c0 + cols, nc);
  }
  const float R = (float)(r + 1);
  int iy, ixl;
  float dy, dxl;
  lin_axis(R, g.y0, g.ysp, g.gny, iy, dy);
  lin_axis((float)(min(c00 + lane, nc - 1) + 1), g.x0, g.xsp, g.gnx, ixl, dxl);
  const int iy2 = g.gny == 1 ? iy : iy + 1;
  const F2 dy2 = both(dy), ey2 = both(FS(1.f, dy)), half = both(0.5f);
  F2 f00 = both(0.f), f01 = f00, f10 = f00, f11 = f00;
  int held = -1;
  for (int c = c0; c < c1; ++c) {  // as many for every lane
    const int ix = __shfl_sync(0xffffffffu, ixl, c - c00);
    const float dx = __shfl_sync(0xffffffffu, dxl, c - c00);
    if (ix != held) {  // uniform, with WRAP within a block
      held = ix;
      const int64_t q0 = (int64_t)ix * g.gny, q1 = (int64_t)(g.gnx == 1 ? ix : ix + 1) * g.gny;
      f00 = pk(pu[iy + q0], pv[iy + q0]);
      f01 = pk(pu[iy + q1], pv[iy + q1]);
      f10 = pk(pu[iy2 + q0], pv[iy2 + q0]);
      f11 = pk(pu[iy2 + q1], pv[iy2 + q1]);
    }
    const F2 dx2 = both(dx), ex2 = both(FS(1.f, dx));
    const F2 a = add2(mul2(ex2, f00), mul2(dx2, f01)), b = add2(mul2(ex2, f10), mul2(dx2, f11));
    float du, dv;  // half the displacement
    unpk(mul2(add2(mul2(ey2, a), mul2(dy2, b)), half), du, dv);
    const float Cc = (float)(c + 1);
    const float ya = FS(R, dv), yb = FA(R, dv), xa = FS(Cc, du), xb = FA(Cc, du);
    bool inya, inyb, inxa, inxb;
    const int iya = spline_cell(ya, nr, inya), iyb = spline_cell(yb, nr, inyb);
    const int ixa = spline_cell(xa, nc, inxa), ixb = spline_cell(xb, nc, inxb);
    const float* ca = CA + (iya - 1) + (ixa - 1) * ld;
    const float* cb = CB + (iyb - 1) + (ixb - 1) * ld;
    F2 wy[4], wx[4], t[4];
    cubw2(mul2, sub2(pk(ya, yb), pk((float)iya, (float)iyb)), wy);
    cubw2(mul2, sub2(pk(xa, xb), pk((float)ixa, (float)ixb)), wx);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const F2 m = mul2(wx[j], pk(__ldg(ca + i + j * ld), __ldg(cb + i + j * ld)));
        t[i] = j == 0 ? m : add2(t[i], m);
      }
    }
    F2 s = mul2(wy[0], t[0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) s = add2(s, mul2(wy[i], t[i]));
    float sa, sb;
    unpk(s, sa, sb);
    if (WRAP ? c < nc : store) {
      const int64_t k = r + (int64_t)c * nr;
      wA[k] = inya && inxa ? sa : 0.f;
      wB[k] = inyb && inxb ? sb : 0.f;
    }
  }
}

template <bool WRAP>
__global__ void __launch_bounds__(256, 3) deform_kernel(const float* __restrict__ CA, const float* __restrict__ CB, int nr,
                                                     int nc, const float* __restrict__ pu,
                                                     const float* __restrict__ pv, PredGrid g, float* wA, float* wB,
                                                        int cols, float minus_zero) {
  const int64_t total = def_strips(WRAP, nr, nc, cols);
  for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < total; k += ((int64_t)gridDim.x * blockDim.x) >> 5)
    deform_strip<WRAP>(CA, CB, nr, nc, pu, pv, g, wA, wB, k, def_cols(WRAP, nr, cols), minus_zero);
}

bool deform_wraps(int64_t nr) { return 4 * 32 * def_row_strips(nr) > 5 * nr; }
int64_t deform_strips(bool wrap, int64_t nr, int64_t nc, int cols) { return def_strips(wrap, nr, nc, cols); }
int deform_cols(const std::function<int64_t(int)>& strips) {
  int cols = DEF_COLS;
  while (cols > 1 && strips(cols) < DEF_STRIPS) cols /= 2;
  return cols;
}

cudaError_t launch_deform(const float* CA, const float* CB, int64_t nr, int64_t nc, const float* pu,
                          const float* pv, PredGrid g, float* wA, float* wB, cudaStream_t s) {
  const bool wrap = deform_wraps(nr);
  const int cols = deform_cols([&](int n) { return def_strips(wrap, nr, nc, n); });
  int64_t blocks = (def_strips(wrap, nr, nc, cols) + 7) / 8;
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (wrap) deform_kernel<true><<<(unsigned)blocks, 256, 0, s>>>(CA, CB, (int)nr, (int)nc, pu, pv, g, wA, wB, cols, -0.0f);
  else deform_kernel<false><<<(unsigned)blocks, 256, 0, s>>>(CA, CB, (int)nr, (int)nc, pu, pv, g, wA, wB, cols, -0.0f);
  return cudaGetLastError();
}

__global__ void node_values_kernel(const float* pu, const float* pv, PredGrid g, const float* y, int32_t ny,
                                   const float* x, int32_t nx, float* u, float* v) {
  const int64_t total = (int64_t)ny * nx;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
    const int gi = (int)(k % ny), gj = (int)(k / ny);
    u[k] = bilinear(pu, g, y[gi], x[gj]);
    v[k] = bilinear(pv, g, y[gi], x[gj]);
  }
}

cudaError_t launch_node_values(const float* pu, const float* pv, PredGrid g, const float* y, int32_t ny,
                               const float* x, int32_t nx, float* u, float* v, cudaStream_t s) {
  const int64_t total = (int64_t)ny * nx;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  node_values_kernel<<<(unsigned)blocks, 256, 0, s>>>(pu, pv, g, y, ny, x, nx, u, v);
  return cudaGetLastError();
}

// ===========================================================================
// Batched forms: every pair of a pass slot in one launch (see hh_batch.h).

#define B_STRIDE(k, n) for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < (n); k += (int64_t)gridDim.x * blockDim.x)

static unsigned b_blocks(int64_t n, int cap_per_sm = 16) {
  int64_t b = (n + 255) / 256;
  if (b > 148 * (int64_t)cap_per_sm) b = 148 * (int64_t)cap_per_sm;
  return (unsigned)(b < 1 ? 1 : b);
}

// prefilter of both frames (blockIdx.y: 0 = A, 1 = B) of every deforming pair.
//
// dim 1 (down the image columns, contiguous in memory) runs on 32-column
// tiles: a warp takes 32 neighbouring columns and one segment, the lanes
// load and store down each column together (coalesced) through a staged
// tile in shared memory, and each lane then runs its own column's sweep
// from the tile with the arithmetic of bs_fwd_item / bs_bwd_item. The
// forward pass reads the image itself (padded element e of column j + 1 is
// image row e - 1), and the backward pass writes every element of the
// padded column, the copied rows 1 and n - 2 included, so no padded copy of
// the image is made first. Work items: (column tile, segment) per pair,
// counted from BPair::wcol.

constexpr int BS_TILE = BS_WARM + BS_SEG;  // rows staged per column
constexpr int BS_TLD = BS_TILE + 1;        // odd stride: conflict-free by lane and by row
constexpr int BSC_WARPS = 4;
constexpr int BS_RPL = (BS_TILE + 31) / 32;  // staged rows per lane and column
// per warp: a tile (32 columns x BS_TILE rows at stride BS_TLD, or BS_TILE
// columns x 32 rows at stride 33) and the elimination factors of its
// BS_TILE unknowns
constexpr int BS_WTILE = BS_TILE * 33 > 32 * BS_TLD ? BS_TILE * 33 : 32 * BS_TLD;
constexpr int BS_WSTRIDE = BS_WTILE + BS_TILE;
constexpr size_t BSC_SMEM = (size_t)BSC_WARPS * BS_WSTRIDE * sizeof(float);

// The factors f[0 .. cnt) into F: every lane of a sweep uses the same factor
// at each step, and staging them keeps an L2 round trip out of the sweep's
// dependent chain. The copies join the tile's asynchronous copies, and
// stage_factors waits for all of them.
__device__ __forceinline__ void bs_cp_async4(float* dst, const float* src);
__device__ __forceinline__ void bs_cp_async_wait_all();
__device__ __forceinline__ void stage_factors(float* F, const float* f, int cnt, int lane) {
  for (int j = lane; j < cnt; j += 32) bs_cp_async4(F + j, f + j);
  bs_cp_async_wait_all();
}

// Rows [0, cnt) (cnt <= BS_TILE) of `ncol` columns between global memory (column
// c at g + c * gld) and a staged tile (column c at T + c * BS_TLD). The
// lanes walk down the columns. Loads are asynchronous copies straight into
// shared memory, all of the tile's issued before the first is waited for (in
// stage_factors): one memory round trip per item instead of one per batch of
// registers.
__device__ __forceinline__ void bs_cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void bs_cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void tile_load(float* T, const float* g, int64_t gld, int ncol, int cnt, int lane) {
  for (int c = 0; c < ncol; ++c)
#pragma unroll
    for (int j = 0; j < BS_RPL; ++j) {
      const int r = lane + 32 * j;
      if (r < cnt) bs_cp_async4(T + c * BS_TLD + r, g + c * gld + r);
    }
}
__device__ __forceinline__ void tile_store(const float* T, float* g, int64_t gld, int ncol, int cnt, int lane) {
  for (int c0 = 0; c0 < ncol; c0 += 8) {
    float v[8][BS_RPL];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < BS_RPL; ++j) {
        const int c = c0 + u, r = lane + 32 * j;
        v[u][j] = (c < ncol && r < cnt) ? T[c * BS_TLD + r] : 0.f;
      }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int j = 0; j < BS_RPL; ++j) {
        const int c = c0 + u, r = lane + 32 * j;
        if (c < ncol && r < cnt) g[c * gld + r] = v[u][j];
      }
  }
}

// Work item l of the column pass of one image (nr x nc, column-major): a
// tile of 32 columns and one segment of their unknowns. coef0 / d0: the
// padded coefficients and the forward-sweep buffer ((nr + 2) x (nc + 2)).
template <int PASS>
__device__ __forceinline__ void bs_col_item(const float* __restrict__ img0, float* coef0, float* d0, int64_t nr,
                                            int64_t nc, const float* __restrict__ cpc, const float* __restrict__ ivc,
                                            int64_t l, float* T, float* F, int lane) {
  {
    const int64_t n = nr + 2, m = n - 4;
    const int64_t ncg = (nc + 31) / 32;
    const int64_t cg = l % ncg, seg = l / ncg;
    const int ncol = (int)min((int64_t)32, nc - cg * 32);  // columns of this tile
    const float* im = img0 + cg * 32 * nr;                     // image column cg*32
    float* coef = coef0 + (cg * 32 + 1) * n;                   // padded column cg*32 + 1
    float* d = d0 + (cg * 32 + 1) * n;
    const bool mine = lane < ncol;
    if (m < 1) {  // n <= 4: nothing to solve; the backward pass writes the column
      if (PASS == 1 && mine) {
        const float* ic = im + lane * nr;
        float* x = coef + lane * n;
        if (n == 4) {
          const float c1 = ic[0], c2 = ic[1];
          x[0] = FS(FM(2.0f, c1), c2);
          x[1] = c1;
          x[2] = c2;
          x[3] = FS(FM(2.0f, c2), c1);
        } else {  // n == 3: the padded copy as it stands
          x[0] = 0.f;
          x[1] = ic[0];
          x[2] = 0.f;
        }
      }
      return;
    }
    const int64_t k0 = seg * BS_SEG, k1 = min(m, k0 + BS_SEG);
    if (PASS == 0) {
      const int64_t ks = max((int64_t)0, k0 - BS_WARM);
      const int cnt = (int)(k1 - ks);
      // stage the right-hand sides: unknown k is padded element k + 2 = image row k + 1
      tile_load(T, im + ks + 1, nr, ncol, cnt, lane);
      stage_factors(F, ivc + ks, cnt, lane);
      __syncwarp();
      if (mine) {
        const float* ic = im + lane * nr;
        const float sixth = kSixth;
        const float c2 = __ldg(ic), cn1 = __ldg(ic + nr - 1);  // padded elements 1 and n - 2
        float* x = T + lane * BS_TLD;
        float dv = 0.f;
#pragma unroll 4
        for (int64_t k = ks; k < k1; ++k) {
          float rhs = x[k - ks];
          if (k == 0) rhs = FS(rhs, FM(sixth, c2));
          if (k == m - 1) rhs = FS(rhs, FM(sixth, cn1));
          dv = k == 0 ? FM(rhs, F[0]) : FM(FS(rhs, FM(sixth, dv)), F[k - ks]);
          x[k - ks] = dv;
        }
      }
      __syncwarp();
      const int nout = (int)(k1 - k0), o = (int)(k0 - ks);
      tile_store(T + o, d + k0 + 2, n, ncol, nout, lane);
      __syncwarp();  // the tile is restaged by the next item
    } else {
      const int64_t ke = min(m - 1, k1 - 1 + BS_WARM);
      const int cnt = (int)(ke - k0 + 1);
      tile_load(T, d + k0 + 2, n, ncol, cnt, lane);
      stage_factors(F, cpc + k0, cnt, lane);
      __syncwarp();
      if (mine) {
        float* x = T + lane * BS_TLD;
        float xv = 0.f, xlast = 0.f;
#pragma unroll 4
        for (int64_t k = ke; k >= k0; --k) {
          const float dk = x[k - k0];
          xv = k == ke ? dk : FS(dk, FM(F[k - k0], xv));
          x[k - k0] = xv;
          if (k == m - 1) xlast = xv;
        }
        const float* ic = im + lane * nr;
        float* xc = coef + lane * n;
        if (k0 == 0) {  // padded element 1 is image row 0; element 0 the "Line" boundary
          const float c1 = __ldg(ic);
          xc[1] = c1;
          xc[0] = FS(FM(2.0f, c1), xv);  // xv == x_0 here
        }
        if (k1 == m) {
          const float cn = __ldg(ic + nr - 1);
          xc[n - 2] = cn;
          xc[n - 1] = FS(FM(2.0f, cn), xlast);
        }
      }
      __syncwarp();
      const int nout = (int)(k1 - k0);
      tile_store(T, coef + k0 + 2, n, ncol, nout, lane);
      __syncwarp();
    }
  }
}

template <int PASS>
__global__ void __launch_bounds__(32 * BSC_WARPS) b_bspline_col_kernel(const BPair* __restrict__ bp, int npairs,
                                                                      int64_t witems, float* dbuf, int64_t qtot) {
  extern __shared__ float bsc_tile[];
  const int img = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* T = bsc_tile + warp * BS_WSTRIDE;
  float* F = T + BS_WTILE;
  for (int64_t t = (int64_t)blockIdx.x * BSC_WARPS + warp; t < witems; t += (int64_t)gridDim.x * BSC_WARPS) {
    const BPair& b = bp[bp_find<&BPair::wcol>(bp, npairs, t)];
    if (!b.deforms) continue;  // uniform across the warp
    const int64_t l = t - b.wcol;
    if (l >= (b.nc + 31) / 32 * b_nseg(b.nr + 2)) continue;
    bs_col_item<PASS>(img ? b.B : b.A, img ? b.coefB : b.coefA, dbuf + (int64_t)img * qtot + b.qoff, b.nr, b.nc,
                      b.cpc, b.ivc, l, T, F, lane);
  }
}

// Padding columns 0 and nc + 1 are written by the row pass's "Line"
// boundary; only rows too short to solve (nc + 2 < 4) keep them zero.
__global__ void b_pad_cols_kernel(const BPair* __restrict__ bp, int npairs) {
  const int img = blockIdx.y;
  for (int p = blockIdx.x; p < npairs; p += gridDim.x) {
    const BPair& b = bp[p];
    if (!b.deforms || b.nc + 2 >= 4) continue;
    const int64_t n = b.nr + 2;
    float* coef = img ? b.coefB : b.coefA;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      coef[i] = 0.f;
      coef[(b.nc + 1) * n + i] = 0.f;
    }
  }
}

// dim 2: a warp takes 32 consecutive padded rows and one segment of their
// unknowns. The segment's columns are staged in shared memory (each column's
// 32 rows are one coalesced 128-byte copy, every column in flight at once),
// the lanes sweep their rows there (row r of staged column j at
// T[33 j + r]: conflict-free), and the results leave the same way. The
// arithmetic is bs_fwd_item / bs_bwd_item's, step for step.
__device__ __forceinline__ void row_tile_load(float* T, const float* g, int64_t gld, int nrow, int cnt, int lane) {
  if (lane < nrow)
    for (int j = 0; j < cnt; ++j) bs_cp_async4(T + j * 33 + lane, g + j * gld + lane);
}
__device__ __forceinline__ void row_tile_store(const float* T, float* g, int64_t gld, int nrow, int cnt, int lane) {
  if (lane >= nrow) return;
  for (int j = 0; j < cnt; ++j) g[j * gld + lane] = T[j * 33 + lane];
}

// Work item l of the row pass of one image's padded coefficients coef0
// ((nr + 2) x (nc + 2)), with the forward-sweep buffer d0 of the same shape.
template <int PASS>
__device__ __forceinline__ void bs_row_item(float* coef0, float* d0, int64_t nr, int64_t nc,
                                            const float* __restrict__ cpr, const float* __restrict__ ivr, int64_t l,
                                            float* T, float* F, int lane) {
  {
    const int64_t ld = nr + 2, n = nc + 2, m = n - 4;
    const int64_t nrg = (ld + 31) / 32;
    const int64_t rg = l % nrg, seg = l / nrg, r0 = rg * 32;
    const int nrow = (int)min((int64_t)32, ld - r0);
    const bool mine = lane < nrow;
    float* coef = coef0 + r0;  // row r0 of the padded coefficients
    float* d = d0 + r0;
    if (PASS == 0) {
      if (m < 1) return;
      const int64_t k0 = seg * BS_SEG, k1 = min(m, k0 + BS_SEG), ks = max((int64_t)0, k0 - BS_WARM);
      const int cnt = (int)(k1 - ks);
      row_tile_load(T, coef + (ks + 2) * ld, ld, nrow, cnt, lane);  // unknown k is padded column k + 2
      stage_factors(F, ivr + ks, cnt, lane);
      __syncwarp();
      if (mine) {
        const float sixth = kSixth;
        const float c2 = coef[ld + lane], cn1 = coef[(n - 2) * ld + lane];
        float dv = 0.f;
#pragma unroll 4
        for (int64_t k = ks; k < k1; ++k) {
          float* x = T + (k - ks) * 33 + lane;
          float rhs = *x;
          if (k == 0) rhs = FS(rhs, FM(sixth, c2));
          if (k == m - 1) rhs = FS(rhs, FM(sixth, cn1));
          dv = k == 0 ? FM(rhs, F[0]) : FM(FS(rhs, FM(sixth, dv)), F[k - ks]);
          *x = dv;
        }
      }
      __syncwarp();
      row_tile_store(T + (k0 - ks) * 33, d + (k0 + 2) * ld, ld, nrow, (int)(k1 - k0), lane);
      __syncwarp();  // the tile is restaged by the next item
    } else {
      if (n < 4) return;
      if (m < 1) {  // n == 4: c1 = b1, c2 = b2 only
        if (mine) {
          const float c1 = coef[ld + lane], c2 = coef[2 * ld + lane];
          coef[lane] = FS(FM(2.0f, c1), c2);
          coef[3 * ld + lane] = FS(FM(2.0f, c2), c1);
        }
        return;
      }
      const int64_t k0 = seg * BS_SEG, k1 = min(m, k0 + BS_SEG), ke = min(m - 1, k1 - 1 + BS_WARM);
      const int cnt = (int)(ke - k0 + 1);
      row_tile_load(T, d + (k0 + 2) * ld, ld, nrow, cnt, lane);
      stage_factors(F, cpr + k0, cnt, lane);
      __syncwarp();
      if (mine) {
        float xv = 0.f, xlast = 0.f;
#pragma unroll 4
        for (int64_t k = ke; k >= k0; --k) {
          float* x = T + (k - k0) * 33 + lane;
          const float dk = *x;
          xv = k == ke ? dk : FS(dk, FM(F[k - k0], xv));
          *x = xv;
          if (k == m - 1) xlast = xv;
        }
        // "Line" boundary columns from the copied columns 1 and n - 2
        if (k0 == 0) coef[lane] = FS(FM(2.0f, coef[ld + lane]), xv);  // xv == x_0 here
        if (k1 == m) coef[(n - 1) * ld + lane] = FS(FM(2.0f, coef[(n - 2) * ld + lane]), xlast);
      }
      __syncwarp();
      row_tile_store(T, coef + (k0 + 2) * ld, ld, nrow, (int)(k1 - k0), lane);
      __syncwarp();
    }
  }
}

template <int PASS>
__global__ void __launch_bounds__(32 * BSC_WARPS) b_bspline_row_kernel(const BPair* __restrict__ bp, int npairs,
                                                                      int64_t witems, float* dbuf, int64_t qtot) {
  extern __shared__ float bsc_tile[];
  const int img = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* T = bsc_tile + warp * BS_WSTRIDE;
  float* F = T + BS_WTILE;
  for (int64_t t = (int64_t)blockIdx.x * BSC_WARPS + warp; t < witems; t += (int64_t)gridDim.x * BSC_WARPS) {
    const BPair& b = bp[bp_find<&BPair::wrow>(bp, npairs, t)];
    if (!b.deforms) continue;  // uniform across the warp
    const int64_t l = t - b.wrow;
    if (l >= (b.nr + 2 + 31) / 32 * b_nseg(b.nc + 2)) continue;
    bs_row_item<PASS>(img ? b.coefB : b.coefA, dbuf + (int64_t)img * qtot + b.qoff, b.nr, b.nc, b.cpr, b.ivr, l, T, F,
                      lane);
  }
}

// The same passes over the two frames of one pair (blockIdx.y: frame), for
// the single-pair schedule and the hooks.
struct PrefFrames {
  const float* img[2];
  float* coef[2];
  float* d[2];
};

template <int PASS>
__global__ void __launch_bounds__(32 * BSC_WARPS) bspline_col_tiles_kernel(PrefFrames P, int64_t nr, int64_t nc,
                                                                          const float* cpc, const float* ivc,
                                                                          int64_t witems) {
  extern __shared__ float bsc_tile[];
  const int img = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* T = bsc_tile + warp * BS_WSTRIDE;
  float* F = T + BS_WTILE;
  for (int64_t t = (int64_t)blockIdx.x * BSC_WARPS + warp; t < witems; t += (int64_t)gridDim.x * BSC_WARPS)
    bs_col_item<PASS>(P.img[img], P.coef[img], P.d[img], nr, nc, cpc, ivc, t, T, F, lane);
}

template <int PASS>
__global__ void __launch_bounds__(32 * BSC_WARPS) bspline_row_tiles_kernel(PrefFrames P, int64_t nr, int64_t nc,
                                                                          const float* cpr, const float* ivr,
                                                                          int64_t witems) {
  extern __shared__ float bsc_tile[];
  const int img = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* T = bsc_tile + warp * BS_WSTRIDE;
  float* F = T + BS_WTILE;
  for (int64_t t = (int64_t)blockIdx.x * BSC_WARPS + warp; t < witems; t += (int64_t)gridDim.x * BSC_WARPS)
    bs_row_item<PASS>(P.coef[img], P.d[img], nr, nc, cpr, ivr, t, T, F, lane);
}

static cudaError_t set_tile_smem() {
  static DeviceOnce done;
  return done([] {
    const auto limit = cudaFuncAttributeMaxDynamicSharedMemorySize;
    for (cudaError_t e : {cudaFuncSetAttribute(b_bspline_col_kernel<0>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(b_bspline_col_kernel<1>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(b_bspline_row_kernel<0>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(b_bspline_row_kernel<1>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(bspline_col_tiles_kernel<0>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(bspline_col_tiles_kernel<1>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(bspline_row_tiles_kernel<0>, limit, (int)BSC_SMEM),
                          cudaFuncSetAttribute(bspline_row_tiles_kernel<1>, limit, (int)BSC_SMEM)})
      if (e != cudaSuccess) return e;
    return cudaSuccess;
  });
}

static unsigned tile_blocks(int64_t witems) {
  int64_t blocks = (witems + BSC_WARPS - 1) / BSC_WARPS;
  if (blocks > 148 * 8) blocks = 148 * 8;
  return (unsigned)(blocks < 1 ? 1 : blocks);
}

cudaError_t launch_prefilter_pair(const float* imgA, const float* imgB, int64_t nr, int64_t nc, float* coefA,
                                  float* coefB, float* dbuf, const float* cpc, const float* ivc, const float* cpr,
                                  const float* ivr, cudaStream_t s) {
  cudaError_t e = set_tile_smem();
  if (e != cudaSuccess) return e;
  const int64_t ld = nr + 2, q = ld * (nc + 2);
  const PrefFrames P{{imgA, imgB}, {coefA, coefB}, {dbuf, dbuf + q}};
  const int64_t wc = (nc + 31) / 32 * b_nseg(ld), wr = (ld + 31) / 32 * b_nseg(nc + 2);
  bspline_col_tiles_kernel<0><<<dim3(tile_blocks(wc), 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(P, nr, nc, cpc, ivc, wc);
  bspline_col_tiles_kernel<1><<<dim3(tile_blocks(wc), 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(P, nr, nc, cpc, ivc, wc);
  if (nc + 2 < 4)  // padding columns 0 and nc + 1 stay zero: no row to solve writes them
    for (float* c : {coefA, coefB}) {
      e = cudaMemsetAsync(c, 0, ld * sizeof(float), s);
      if (e == cudaSuccess) e = cudaMemsetAsync(c + (nc + 1) * ld, 0, ld * sizeof(float), s);
      if (e != cudaSuccess) return e;
    }
  bspline_row_tiles_kernel<0><<<dim3(tile_blocks(wr), 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(P, nr, nc, cpr, ivr, wr);
  bspline_row_tiles_kernel<1><<<dim3(tile_blocks(wr), 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(P, nr, nc, cpr, ivr, wr);
  return cudaGetLastError();
}

cudaError_t launch_b_prefilter(const BPair* bp, int npairs, int64_t qtot, int64_t wcol_tot, int64_t wrow_tot,
                               float* dbuf, cudaStream_t s) {
  if (qtot <= 0) return cudaSuccess;
  cudaError_t e = set_tile_smem();
  if (e != cudaSuccess) return e;
  if (wcol_tot > 0) {
    int64_t blocks = (wcol_tot + BSC_WARPS - 1) / BSC_WARPS;
    if (blocks > 148 * 8) blocks = 148 * 8;
    b_bspline_col_kernel<0><<<dim3((unsigned)blocks, 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(bp, npairs, wcol_tot, dbuf, qtot);
    b_bspline_col_kernel<1><<<dim3((unsigned)blocks, 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(bp, npairs, wcol_tot, dbuf, qtot);
  }
  b_pad_cols_kernel<<<dim3(npairs < 148 ? npairs : 148, 2), 128, 0, s>>>(bp, npairs);
  if (wrow_tot > 0) {
    int64_t blocks = (wrow_tot + BSC_WARPS - 1) / BSC_WARPS;
    if (blocks > 148 * 8) blocks = 148 * 8;
    b_bspline_row_kernel<0><<<dim3((unsigned)blocks, 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(bp, npairs, wrow_tot, dbuf, qtot);
    b_bspline_row_kernel<1><<<dim3((unsigned)blocks, 2), 32 * BSC_WARPS, BSC_SMEM, s>>>(bp, npairs, wrow_tot, dbuf, qtot);
  }
  return cudaGetLastError();
}

// the predictor grid of sweep `it`: the previous slot's grid in sweep 1,
// this slot's grid afterwards
__device__ __forceinline__ PredGrid b_pred_grid(const BPair& b, int it) {
  PredGrid g;
  if (it == 1) {
    g.gny = b.pgny; g.gnx = b.pgnx; g.y0 = b.py0; g.ysp = b.pysp; g.x0 = b.px0; g.xsp = b.pxsp;
  } else {
    g.gny = b.ny; g.gnx = b.nx; g.y0 = b.gy0; g.ysp = b.gysp; g.x0 = b.gx0; g.xsp = b.gxsp;
  }
  return g;
}

// Start of sweep `it`: the node values of the predictor (zero without one),
// NaN uncertainties at the start of the slot, and the sweep count of pairs
// in their final pass.
__global__ void b_sweep_begin_kernel(const BPair* __restrict__ bp, int npairs, const int32_t* __restrict__ done, int it,
                                     int64_t gtot, const float* __restrict__ pu, const float* __restrict__ pv, float* u,
                                     float* v, float* uncu, float* uncv, int32_t* sweeps, int32_t* slot_sweeps) {
  B_STRIDE(k, gtot) {
    const int p = bp_find<&BPair::coff>(bp, npairs, k);
    const BPair& b = bp[p];
    const int64_t l = k - b.coff;
    if (!bp_live(b, it, done, p) || l >= (int64_t)b.ny * b.nx) continue;
    const int64_t id = b.goff + l;
    if (l == 0) {
      slot_sweeps[p] = it;
      if (b.is_final) sweeps[p] = it;
    }
    if (it == 1) {
      uncu[id] = __int_as_float(0x7fc00000);
      uncv[id] = __int_as_float(0x7fc00000);
    }
    if (it > 1 || b.has_pred0) {
      const PredGrid g = b_pred_grid(b, it);
      const int gi = (int)(l % b.ny), gj = (int)(l / b.ny);
      const float y = FA(b.gy0, FM((float)gi, b.gysp)), x = FA(b.gx0, FM((float)gj, b.gxsp));
      u[id] = bilinear(pu + b.goff, g, y, x);
      v[id] = bilinear(pv + b.goff, g, y, x);
    } else {
      u[id] = 0.f;
      v[id] = 0.f;
    }
  }
}

cudaError_t launch_b_sweep_begin(const BPair* bp, int npairs, const int32_t* done, int it, int64_t gtot,
                                 const float* pu, const float* pv, float* u, float* v, float* uncu, float* uncv,
                                 int32_t* sweeps, int32_t* slot_sweeps, cudaStream_t s) {
  if (gtot <= 0) return cudaSuccess;
  b_sweep_begin_kernel<<<b_blocks(gtot), 256, 0, s>>>(bp, npairs, done, it, gtot, pu, pv, u, v, uncu, uncv, sweeps,
                                                      slot_sweeps);
  return cudaGetLastError();
}

// Strips (deform_strip) of every pair that deforms, a warp each; the pair of a
// strip is looked up once.
template <bool WRAP>
__global__ void __launch_bounds__(256, 3) b_deform_kernel(const BPair* __restrict__ bp, int npairs,
                                                       const int32_t* __restrict__ done, int it, int64_t stot, int cols,
                                                       const float* __restrict__ pu, const float* __restrict__ pv, float minus_zero) {
  for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < stot; k += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int p = bp_find<&BPair::dcoff>(bp, npairs, k);
    const BPair& b = bp[p];
    if (!bp_live(b, it, done, p) || !(it > 1 || b.has_pred0) || !b.deforms) continue;  // uniform across the warp
    deform_strip<WRAP>(b.coefA, b.coefB, (int)b.nr, (int)b.nc, pu + b.goff, pv + b.goff, b_pred_grid(b, it), b.warpA, b.warpB,
                       k - b.dcoff, def_cols(WRAP, b.nr, cols), minus_zero);
  }
}

cudaError_t launch_b_deform(const BPair* bp, int npairs, const int32_t* done, int it, int64_t stot, bool wrap, int cols,
                            const float* pu, const float* pv, cudaStream_t s) {
  if (stot <= 0) return cudaSuccess;
  const unsigned blocks = b_blocks(stot * 32, 32);
  if (wrap) b_deform_kernel<true><<<blocks, 256, 0, s>>>(bp, npairs, done, it, stot, cols, pu, pv, -0.0f);
  else b_deform_kernel<false><<<blocks, 256, 0, s>>>(bp, npairs, done, it, stot, cols, pu, pv, -0.0f);
  return cudaGetLastError();
}

}  // namespace hh
