// Vector-grid kernels of a WIDIM sweep on one image pair (sm_100a):
// combine, validation, peak substitution, replacement, predictor
// smoothing, convergence norm. The per-cell logic lives in hh_grid.cuh.
#include <math.h>
#include <stdint.h>

#include "hh_grid.cuh"
#include "hh_internal.h"
#include "hh_pred.cuh"

namespace hh {

static inline int grid_blocks(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

#define GRID_STRIDE(k, n) for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < (n); k += (int64_t)gridDim.x * blockDim.x)

// u = predictor + residual, alternatives + predictor, masked -> NaN
// (src/pipeline.jl:755-767), optional measured copy (:768-770). The
// predictor's node value is formed here, at node (y0 + i ysp, x0 + j xsp)
// (0 without a predictor).
__global__ void combine_kernel(float* u, float* v, const float* resu, const float* resv, float* ratio, float* moment,
                               float* alt_u, float* alt_v, int32_t nalt, const uint8_t* gmask, int32_t ny, int32_t nx,
                               NodePred pr, float* meas_u, float* meas_v) {
  const int64_t G = (int64_t)ny * nx;
  GRID_STRIDE(k, G) {
    float pu = 0.f, pv = 0.f;
    if (pr.u) {
      const float y = FA(pr.y0, FM((float)(k % ny), pr.ysp)), x = FA(pr.x0, FM((float)(k / ny), pr.xsp));
      pu = bilinear(pr.u, pr.g, y, x);
      pv = bilinear(pr.v, pr.g, y, x);
    }
    for (int m = 0; m < nalt; ++m) {
      alt_u[k + m * G] = FADD(alt_u[k + m * G], pu);
      alt_v[k + m * G] = FADD(alt_v[k + m * G], pv);
    }
    float uu = FADD(pu, resu[k]), vv = FADD(pv, resv[k]);
    if (gmask && gmask[k]) {
      uu = vv = f_nan();
      ratio[k] = f_nan();
      moment[k] = f_nan();
    }
    u[k] = uu;
    v[k] = vv;
    if (meas_u) {
      meas_u[k] = uu;
      meas_v[k] = vv;
    }
  }
}

cudaError_t launch_combine(float* u, float* v, const float* resu, const float* resv, float* ratio, float* moment,
                           float* alt_u, float* alt_v, int32_t nalt, const uint8_t* gmask, int32_t ny, int32_t nx,
                           const NodePred& pr, float* meas_u, float* meas_v, cudaStream_t s) {
  combine_kernel<<<grid_blocks((int64_t)ny * nx), 256, 0, s>>>(u, v, resu, resv, ratio, moment, alt_u, alt_v, nalt,
                                                               gmask, ny, nx, pr, meas_u, meas_v);
  return cudaGetLastError();
}

__global__ void uod_kernel(const float* u, const float* v, int32_t ny, int32_t nx, double thr, int32_t nb, double eps,
                           const uint8_t* exclude, uint8_t* flags, int32_t or_into) {
  GRID_STRIDE(k, (int64_t)ny * nx) {
    const uint8_t f = uod_cell(u, v, ny, nx, (int)(k % ny), (int)(k / ny), thr, nb, eps, exclude);
    if (or_into) flags[k] |= f;
    else flags[k] = f;
  }
}

cudaError_t launch_uod(const float* u, const float* v, int32_t ny, int32_t nx, double thr, int32_t nb, double eps,
                       const uint8_t* exclude, uint8_t* flags, int32_t or_into, cudaStream_t s) {
  if (nb < 1 || (2 * nb + 1) * (2 * nb + 1) - 1 > UOD_MAXN) return cudaErrorInvalidValue;
  uod_kernel<<<grid_blocks((int64_t)ny * nx, 128), 128, 0, s>>>(u, v, ny, nx, thr, nb, eps, exclude, flags, or_into);
  return cudaGetLastError();
}

// validate_and_replace!'s flags in one pass (src/pipeline.jl:617-645,
// apply_validator! src/quality.jl:466-486): the outlier detection, the peak
// ratio and the extra validators; masked cells cleared. Written twice: the
// snapshot that the substitution judges by, and the flags it updates.
__global__ void __launch_bounds__(128, 4) flags_kernel(const float* u, const float* v, const float* ratio, const float* moment, int32_t ny,
                             int32_t nx, FlagRules r, const uint8_t* gmask, uint8_t* flags, uint8_t* flags2) {
  GRID_STRIDE(k, (int64_t)ny * nx) {
    uint8_t f = 0;
    if (!(gmask && gmask[k])) {
      const int gi = (int)(k % ny), gj = (int)(k / ny);
      if (r.min_ratio > 1 && !((double)ratio[k] >= r.min_ratio)) f = 1;
      // the detection as rule -1 among the extra validators, so that its code is
      // there once, and 128 registers: twice took 203, too many for the local
      // arrays of 3 and 4 layers (500 x 400 cells: 1806 and 5588 us instead of
      // 1098 and 3754; 2 layers 35 and 37)
#pragma unroll 1
      for (int q = r.uod ? -1 : 0; q < r.nval; ++q) {
        const hh_validator vd = q < 0 ? hh_validator{HH_VAL_UOD, r.uod_nb, r.uod_thr, 0, 0, 0.1} : r.val[q];
        if (vd.kind == HH_VAL_PEAK_RATIO) {
          if (!((double)ratio[k] >= vd.threshold)) f = 1;
        } else if (vd.kind == HH_VAL_MOMENT) {
          if (!((double)moment[k] <= vd.threshold)) f = 1;
        } else if (vd.kind == HH_VAL_VELOCITY) {
          const double mag = (double)hypotf(u[k], v[k]);
          if (!(vd.vmin <= mag && mag <= vd.vmax)) f = 1;
        } else if (vd.kind == HH_VAL_UOD) {
          f |= uod_cell(u, v, ny, nx, gi, gj, vd.threshold, vd.neighborhood, vd.epsilon, gmask);
        }
      }
    }
    flags[k] = f;
    if (flags2) flags2[k] = f;
  }
}
cudaError_t launch_flags(const float* u, const float* v, const float* ratio, const float* moment, int32_t ny, int32_t nx,
                         const FlagRules& r, const uint8_t* gmask, uint8_t* flags, uint8_t* flags2, cudaStream_t s) {
  auto served = [](int nb) { return nb >= 1 && (2 * nb + 1) * (2 * nb + 1) - 1 <= UOD_MAXN; };
  if (r.uod && !served(r.uod_nb)) return cudaErrorInvalidValue;
  for (int q = 0; q < r.nval; ++q)
    if (r.val[q].kind == HH_VAL_UOD && !served(r.val[q].neighborhood)) return cudaErrorInvalidValue;
  flags_kernel<<<grid_blocks((int64_t)ny * nx, 128), 128, 0, s>>>(u, v, ratio, moment, ny, nx, r, gmask, flags, flags2);
  return cudaGetLastError();
}

template <bool WIDE>
__global__ void __launch_bounds__(128, WIDE ? 12 : 3)
    substitute_kernel(float* u, float* v, const uint8_t* outl_in, uint8_t* outl_out, const uint8_t* gmask,
                      const float* alt_u, const float* alt_v, int32_t nalt, int32_t ny, int32_t nx, int32_t er,
                      double thr) {
  GRID_STRIDE(k, (int64_t)ny * nx)
  outl_out[k] = substitute_cell<WIDE>(u, v, outl_in, gmask, alt_u, alt_v, nalt, ny, nx, (int)(k % ny), (int)(k / ny), er, thr);
}

cudaError_t launch_substitute(float* u, float* v, const uint8_t* outl_in, uint8_t* outl_out, const uint8_t* gmask,
                              const float* alt_u, const float* alt_v, int32_t nalt, int32_t ny, int32_t nx, int32_t er,
                              double thr, cudaStream_t s) {
  if (er < 1 || (2 * er + 1) * (2 * er + 1) - 1 > UOD_MAXN) return cudaErrorInvalidValue;
  const int blocks = grid_blocks((int64_t)ny * nx, 128);
  if (er > 2) substitute_kernel<true><<<blocks, 128, 0, s>>>(u, v, outl_in, outl_out, gmask, alt_u, alt_v, nalt, ny, nx, er, thr);
  else substitute_kernel<false><<<blocks, 128, 0, s>>>(u, v, outl_in, outl_out, gmask, alt_u, alt_v, nalt, ny, nx, er, thr);
  return cudaGetLastError();
}

__global__ void replace_kernel(float* u, float* v, const uint8_t* flags, const uint8_t* gmask, int32_t ny, int32_t nx,
                               int32_t nan_mask) {
  GRID_STRIDE(k, (int64_t)ny * nx) {
    if (!repl_invalid(flags, gmask, k)) continue;
    float nu = u[k], nvv = v[k];
    // a masked cell that ends as NaN is not searched for (no other cell reads it)
    if (nan_mask && gmask && gmask[k]) nu = nvv = f_nan();
    else replace_cell(u, v, flags, gmask, ny, nx, (int)(k % ny), (int)(k / ny), nu, nvv);
    u[k] = nu;
    v[k] = nvv;
  }
}

cudaError_t launch_replace(float* u, float* v, const uint8_t* flags, const uint8_t* gmask, int32_t ny, int32_t nx,
                           int32_t nan_mask, cudaStream_t s) {
  replace_kernel<<<grid_blocks((int64_t)ny * nx, 128), 128, 0, s>>>(u, v, flags, gmask, ny, nx, nan_mask);
  return cudaGetLastError();
}

__global__ void smooth_kernel(const float* f, int32_t ny, int32_t nx, float* out) {
  GRID_STRIDE(k, (int64_t)ny * nx) out[k] = smooth_cell(f, ny, nx, (int)(k % ny), (int)(k / ny));
}
cudaError_t launch_smooth(const float* f, int32_t ny, int32_t nx, float* out, cudaStream_t s) {
  smooth_kernel<<<grid_blocks((int64_t)ny * nx), 256, 0, s>>>(f, ny, nx, out);
  return cudaGetLastError();
}

// build_predictor (src/pipeline.jl:454-464) from the validated field (u, v):
// masked cells from their valid neighbours into (wu, wv) when there is a mask,
// then the [1 2 1] smoothing into (ou, ov); with prev_u, the field is also
// kept for the next sweep's convergence test.
__global__ void pred_fill_kernel(const float* u, const float* v, const uint8_t* gmask, int32_t ny, int32_t nx,
                                 float* wu, float* wv) {
  GRID_STRIDE(k, (int64_t)ny * nx) {
    float nu = u[k], nv = v[k];
    if (gmask && gmask[k]) replace_cell(u, v, nullptr, gmask, ny, nx, (int)(k % ny), (int)(k / ny), nu, nv);
    wu[k] = nu;
    wv[k] = nv;
  }
}
__global__ void pred_smooth_kernel(const float* u, const float* v, int32_t ny, int32_t nx, float* ou, float* ov,
                                   const float* cur_u, const float* cur_v, float* prev_u, float* prev_v) {
  GRID_STRIDE(k, (int64_t)ny * nx) {
    if (ou) {
      ou[k] = smooth_cell(u, ny, nx, (int)(k % ny), (int)(k / ny));
      ov[k] = smooth_cell(v, ny, nx, (int)(k % ny), (int)(k / ny));
    }
    if (prev_u) {
      prev_u[k] = cur_u[k];
      prev_v[k] = cur_v[k];
    }
  }
}
cudaError_t launch_predictor(const float* u, const float* v, const uint8_t* gmask, int32_t ny, int32_t nx, bool smoothing,
                             float* wu, float* wv, float* ou, float* ov, float* prev_u, float* prev_v, cudaStream_t s) {
  const int64_t G = (int64_t)ny * nx;
  const bool fill = gmask || !smoothing;
  if (fill) pred_fill_kernel<<<grid_blocks(G, 128), 128, 0, s>>>(u, v, gmask, ny, nx, wu, wv);
  if (smoothing || prev_u)
    pred_smooth_kernel<<<grid_blocks(G), 256, 0, s>>>(fill ? wu : u, fill ? wv : v, ny, nx, smoothing ? ou : nullptr,
                                                      smoothing ? ov : nullptr, u, v, prev_u, prev_v);
  return cudaGetLastError();
}

// The window list of an unmasked grid, column-major grid order: 4 int32 per
// window (gi, gj, rs, cs).
__global__ void make_jobs_kernel(int4* jobs, int32_t ny, int64_t G, WinGrid w) {
  GRID_STRIDE(k, G) {
    const int gi = (int)(k % ny), gj = (int)(k / ny);
    jobs[k] = make_int4(gi, gj, w.r0 + gi * w.rstep, w.c0 + gj * w.cstep);
  }
}
cudaError_t launch_make_jobs(int32_t* jobs, int32_t ny, int32_t nx, const WinGrid& w, cudaStream_t s) {
  const int64_t G = (int64_t)ny * nx;
  make_jobs_kernel<<<grid_blocks(G), 256, 0, s>>>(reinterpret_cast<int4*>(jobs), ny, G, w);
  return cudaGetLastError();
}

// Grid mask (pass_grid, src/pipeline.jl:529-555): a window whose masked
// fraction, of the window or of its search area, reaches thr. A warp a window.
__global__ void mask_grid_kernel(const uint8_t* mask, int64_t nr, int32_t ny, int64_t G, WinGrid w, int32_t wr, int32_t wc,
                                 int32_t mr, int32_t mc, double thr, uint8_t* gmask) {
  const int lane = threadIdx.x & 31;
  for (int64_t k = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); k < G;
       k += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const int64_t rs = w.r0 + (k % ny) * w.rstep, cs = w.c0 + (k / ny) * w.cstep;  // the window's first pixel
    int cw = 0, ca = 0;
    for (int j = -mc; j < wc + mc; ++j)
      for (int i = -mr + lane; i < wr + mr; i += 32) {
        const int m = mask[(rs + i) + (cs + j) * nr] != 0;
        ca += m;
        cw += (i >= 0 && i < wr && j >= 0 && j < wc) ? m : 0;
      }
    cw = __reduce_add_sync(0xffffffffu, cw);
    ca = __reduce_add_sync(0xffffffffu, ca);
    if (lane == 0) {
      const double fw = (double)cw / (double)(wr * wc), fs = (double)ca / (double)((wr + 2 * mr) * (wc + 2 * mc));
      gmask[k] = fw >= thr || fs >= thr;
    }
  }
}
cudaError_t launch_mask_grid(const uint8_t* mask, int64_t nr, int32_t ny, int32_t nx, const WinGrid& w, int32_t wr,
                             int32_t wc, int32_t mr, int32_t mc, double thr, uint8_t* gmask, cudaStream_t s) {
  const int64_t G = (int64_t)ny * nx;
  mask_grid_kernel<<<grid_blocks(G, 4), 128, 0, s>>>(mask, nr, ny, G, w, wr, wc, mr, mc, thr, gmask);
  return cudaGetLastError();
}

// field_change (src/pipeline.jl:849-866): one cluster, keys in scratch.
__global__ void __cluster_dims__(FC_CLUSTER, 1, 1) __launch_bounds__(FC_THREADS)
    field_change_kernel(const float* u, const float* v, const float* pu, const float* pv, const uint8_t* gmask,
                        int64_t G, uint32_t* keys, float* out) {
  __shared__ FieldChangeSmem sm;
  const float change = cluster_field_change(sm, G, keys, [&](int64_t i, bool& counts) {
    return change_key(u[i], v[i], pu[i], pv[i], gmask && gmask[i], counts);
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) *out = change;
}

cudaError_t launch_field_change(const float* u, const float* v, const float* pu, const float* pv, const uint8_t* gmask,
                                int64_t G, float* scratch, float* out, cudaStream_t s) {
  field_change_kernel<<<FC_CLUSTER, FC_THREADS, 0, s>>>(u, v, pu, pv, gmask, G, reinterpret_cast<uint32_t*>(scratch),
                                                        out);
  return cudaGetLastError();
}

__global__ void restore_measured_kernel(float* u, float* v, const float* mu, const float* mv, const uint8_t* outl,
                                        int64_t G) {
  GRID_STRIDE(k, G) if (outl[k]) {
    u[k] = mu[k];
    v[k] = mv[k];
  }
}
cudaError_t launch_restore_measured(float* u, float* v, const float* meas_u, const float* meas_v, const uint8_t* outl,
                                    int64_t G, cudaStream_t s) {
  restore_measured_kernel<<<grid_blocks(G), 256, 0, s>>>(u, v, meas_u, meas_v, outl, G);
  return cudaGetLastError();
}

__global__ void fill_kernel(float* p, float value, int64_t n) {
  GRID_STRIDE(k, n) p[k] = value;
}
cudaError_t launch_fill(float* p, float value, int64_t n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  fill_kernel<<<grid_blocks(n), 256, 0, s>>>(p, value, n);
  return cudaGetLastError();
}

}  // namespace hh
