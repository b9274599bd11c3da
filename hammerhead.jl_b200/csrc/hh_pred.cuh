// The WIDIM predictor: bilinear interpolation on a uniform node grid with
// flat extrapolation (Gridded(Linear()) + Flat(), src/pipeline.jl:561-600),
// in explicit round-to-nearest arithmetic.
#pragma once
#include "hh_internal.h"

namespace hh {

#define FM(a, b) __fmul_rn((a), (b))
#define FA(a, b) __fadd_rn((a), (b))
#define FS(a, b) __fsub_rn((a), (b))
#define FD(a, b) __fdiv_rn((a), (b))

// Gridded(Linear()) + Flat() along one axis of uniform knots q0 + k*step.
__device__ __forceinline__ void lin_axis(float q, float q0, float step, int n, int& i, float& d) {
  if (n == 1) { i = 0; d = 0.f; return; }
  const float last = FA(q0, FM((float)(n - 1), step));
  if (q <= q0) { i = 0; d = 0.f; return; }
  if (q >= last) { i = n - 2; d = 1.f; return; }
  i = (int)floorf(FD(FS(q, q0), step));
  if (i > n - 2) i = n - 2;
  const float k0 = FA(q0, FM((float)i, step)), k1 = FA(q0, FM((float)(i + 1), step));
  d = FD(FS(q, k0), FS(k1, k0));
}

__device__ __forceinline__ float bilinear(const float* f, const PredGrid& g, float qy, float qx) {
  int iy, ix;
  float dy, dx;
  lin_axis(qy, g.y0, g.ysp, g.gny, iy, dy);
  lin_axis(qx, g.x0, g.xsp, g.gnx, ix, dx);
  const int iy2 = g.gny == 1 ? iy : iy + 1, ix2 = g.gnx == 1 ? ix : ix + 1;
  const float f00 = f[iy + ix * g.gny], f01 = f[iy + ix2 * g.gny], f10 = f[iy2 + ix * g.gny],
              f11 = f[iy2 + ix2 * g.gny];
  const float a = FA(FM(FS(1.f, dx), f00), FM(dx, f01));
  const float b = FA(FM(FS(1.f, dx), f10), FM(dx, f11));
  return FA(FM(FS(1.f, dy), a), FM(dy, b));
}

}  // namespace hh
