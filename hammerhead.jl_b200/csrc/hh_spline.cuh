// The division by 6 of the cubic B-spline weights, shared by the deformation
// and its adjoint.
#pragma once
#include <cuda_runtime.h>

namespace hh {

// x / 6 correctly rounded for every x whose quotient is a normal float (and
// x = 0), without a division: q0 = x * RN(1/6), then one residual correction
// by fused multiply-add (Markstein's correction for a divisor known in
// advance; Brisebarre, Muller and Raina, IEEE Trans. Computers 53(8), 2004).
// A comparison with IEEE division over every positive float with a normal
// quotient finds no difference. The B-spline weights (1-d)^3 and d^3 it
// divides are 0 or at least 2^-72 (d is 0 or a multiple of 2^-23 in [0, 1]),
// so their quotients are normal.
static __device__ __forceinline__ float div6(float x) {
  const float r = __int_as_float(0x3E2AAAAB);  // 1/6 rounded
  const float q0 = __fmul_rn(x, r);
  const float e = __fmaf_rn(-q0, 6.0f, x);
  return __fmaf_rn(e, r, q0);
}

}  // namespace hh
