// Ensemble (sum-of-correlation) PIV on the device: run_piv_ensemble
// (src/ensemble.jl:51-205). Per pass, every pair is staged and deformed by
// the shared predictor, the correlation kernel adds each window's plane to a
// device-resident accumulator (and the Wieneke statistics to FP64 sums), and
// after the last pair the summed planes are analysed once, combined with the
// predictor and validated exactly like a WIDIM sweep. Only the final vector
// grid returns to the host. With the pairs split over processes, the context
// reducer (hh_set_ensemble_reducer) turns each pass's partial sums into the
// sums over all processes before the analysis.
#include "hh_ctx.h"

using namespace hhd;

extern "C" hh_status hh_run_ensemble(hh_ctx* ctx, const hh_batch_pair* pairs, int32_t npairs,
                                     const hh_pass_desc* passes, int32_t np, const uint8_t* hmask, double thr,
                                     int32_t smoothing, int32_t flags, hh_result* out) {
  if (!ctx) return fail(nullptr, HH_ERR_ARG, "context is NULL");
  HH_TRY(set_device(ctx));
  if (!pairs || npairs < 1) return fail(ctx, HH_ERR_ARG, "pairs must not be empty");
  HH_TRY(check_passes(ctx, passes, np));
  if (!(thr > 0 && thr <= 1)) return fail(ctx, HH_ERR_ARG, "mask_threshold must be in (0, 1], got " + num(thr));
  const int64_t nr = pairs[0].nr, nc = pairs[0].nc, P = nr * nc;
  if (nr < 1 || nc < 1) return fail(ctx, HH_ERR_ARG, "images must be non-empty");
  for (int q = 0; q < npairs; ++q) {
    if (pairs[q].nr != nr || pairs[q].nc != nc)
      return fail(ctx, HH_ERR_ARG, "all pairs must share the image size (" + std::to_string(nr) + ", " +
                                       std::to_string(nc) + "), got (" + std::to_string(pairs[q].nr) + ", " +
                                       std::to_string(pairs[q].nc) + ")");
    if (!pairs[q].A || !pairs[q].B) return fail(ctx, HH_ERR_ARG, "image pointer is NULL");
    if (pairs[q].format < HH_PIX_F32 || pairs[q].format > HH_PIX_U16_RAW)
      return fail(ctx, HH_ERR_ARG, "unknown pixel format " + std::to_string(pairs[q].format));
  }
  const bool device_inputs = (flags & HH_BATCH_DEVICE_INPUTS) != 0;
  cudaStream_t s = ctx->stream;
  uint8_t* dmask = nullptr;
  if (hmask) {
    HH_TRY(buf(ctx, "ens_mask", (size_t)P, &dmask));
    HH_CK(cudaMemcpyAsync(dmask, hmask, (size_t)P, cudaMemcpyHostToDevice, s));
  }
  std::vector<Grid> grids;
  HH_TRY(pass_grids(ctx, nr, nc, passes, np, dmask, thr, grids));
  int64_t Gmax = 1, Jmax = 1, accmax = 1;
  int nalt_max = 0;
  for (int k = 0; k < np; ++k) {
    const int64_t nj = grid_njobs(grids[k]);
    const int64_t PL = (int64_t)fft_rows(passes[k]) * fft_cols(passes[k]);
    Gmax = std::max<int64_t>(Gmax, grids[k].G());
    Jmax = std::max<int64_t>(Jmax, nj);
    accmax = std::max<int64_t>(accmax, nj * PL);
    nalt_max = std::max(nalt_max, passes[k].n_peaks - 1);
  }
  float *dA = nullptr, *dB = nullptr, *coefA, *coefB, *warpA, *warpB, *acc;
  double* stats;
  bool any_u16 = false;
  for (int q = 0; q < npairs; ++q) any_u16 |= pairs[q].format != HH_PIX_F32;
  uint16_t *d16A = nullptr, *d16B = nullptr;
  if (!device_inputs || any_u16) {
    HH_TRY(buf(ctx, "ens_A", (size_t)P, &dA));
    HH_TRY(buf(ctx, "ens_B", (size_t)P, &dB));
  }
  if (!device_inputs && any_u16) {
    HH_TRY(buf(ctx, "ens_A16", (size_t)P, &d16A));
    HH_TRY(buf(ctx, "ens_B16", (size_t)P, &d16B));
  }
  HH_TRY(buf(ctx, "coefA", (size_t)(nr + 2) * (nc + 2), &coefA));
  HH_TRY(buf(ctx, "coefB", (size_t)(nr + 2) * (nc + 2), &coefB));
  HH_TRY(buf(ctx, "warpA", (size_t)P, &warpA));
  HH_TRY(buf(ctx, "warpB", (size_t)P, &warpB));
  HH_TRY(buf(ctx, "ens_acc", (size_t)accmax, &acc));
  HH_TRY(buf(ctx, "ens_stats", (size_t)Jmax * 88, &stats));
  ResultBlock rb;
  HH_TRY(result_block(ctx, Gmax, rb));
  float *u = rb.u, *v = rb.v, *ratio = rb.ratio, *moment = rb.moment, *uncu = rb.uncu, *uncv = rb.uncv;
  uint8_t* outl = rb.outl;
  float *resu, *resv, *altu = nullptr, *altv = nullptr, *predu, *predv, *predw_u, *predw_v;
  uint8_t *outl2, *gm;
  int32_t* djobs;
  HH_TRY(buf(ctx, "resu", Gmax, &resu));
  HH_TRY(buf(ctx, "resv", Gmax, &resv));
  if (nalt_max > 0) {
    HH_TRY(buf(ctx, "altu", Gmax * nalt_max, &altu));
    HH_TRY(buf(ctx, "altv", Gmax * nalt_max, &altv));
  }
  HH_TRY(buf(ctx, "predu", Gmax, &predu));
  HH_TRY(buf(ctx, "predv", Gmax, &predv));
  HH_TRY(buf(ctx, "predwu", Gmax, &predw_u));
  HH_TRY(buf(ctx, "predwv", Gmax, &predw_v));
  HH_TRY(buf(ctx, "outl2", Gmax, &outl2));
  HH_TRY(buf(ctx, "gmask", Gmax, &gm));
  HH_TRY(buf(ctx, "jobs", 4 * Jmax, &djobs));
  while ((int)ctx->events.size() < np + 1) {
    cudaEvent_t e;
    HH_CK(cudaEventCreate(&e));
    ctx->events.push_back(e);
  }
  ctx->pass_ms.assign(np, 0.f);
  ctx->pass_sweeps.assign(np, 1);
  HH_CK(cudaEventRecord(ctx->events[0], s));

  const float NaN = std::nanf("");
  hh::PredGrid pg{};
  const float* pred_src_u = nullptr;
  const float* pred_src_v = nullptr;
  for (int k = 0; k < np; ++k) {
    const hh_pass_desc& p = passes[k];
    const Grid& g = grids[k];
    const bool force_replace = k < np - 1;
    const int ny = g.ny, nx = g.nx;
    const int64_t G = (int64_t)ny * nx;
    const int64_t njobs = grid_njobs(g);
    const int W = p.window[0], NR = fft_rows(p), NC = fft_cols(p);
    const int64_t PL = (int64_t)NR * NC;
    const int nalt = p.n_peaks - 1;
    const bool unc = p.uncertainty && !force_replace;
    Tables tb;
    HH_TRY(get_tables(ctx, p, tb));
    if (k > 0) {  // build_predictor from the previous pass's result (src/pipeline.jl:454-464)
      const Grid& pgd = grids[k - 1];
      HH_K(HH_K_VECTOR, hh::predictor_launches(pgd.any_mask, smoothing, false), 0, 24 * pgd.G(), pgd.G(),
           hh::launch_predictor(u, v, pgd.any_mask ? gm : nullptr, pgd.ny, pgd.nx, smoothing, predw_u, predw_v, predu, predv,
                                nullptr, nullptr, s));
      pred_src_u = smoothing ? predu : predw_u;
      pred_src_v = smoothing ? predv : predw_v;
      pg = pred_grid(pgd);
    }
    HH_TRY(stage_grid(ctx, g, djobs, gm));
    HH_CK(cudaMemsetAsync(acc, 0, (size_t)njobs * PL * sizeof(float), s));
    if (unc) HH_CK(cudaMemsetAsync(stats, 0, (size_t)njobs * 88 * sizeof(double), s));
    for (int q = 0; q < npairs; ++q) {
      const float* A = pairs[q].A;
      const float* B = pairs[q].B;
      if (pairs[q].format != HH_PIX_F32) {  // UInt16 frames: (copy and) convert on the device
        const uint16_t* a16 = reinterpret_cast<const uint16_t*>(A);
        const uint16_t* b16 = reinterpret_cast<const uint16_t*>(B);
        if (!device_inputs) {
          HH_CK(cudaMemcpyAsync(d16A, a16, P * sizeof(uint16_t), cudaMemcpyHostToDevice, s));
          HH_CK(cudaMemcpyAsync(d16B, b16, P * sizeof(uint16_t), cudaMemcpyHostToDevice, s));
          a16 = d16A;
          b16 = d16B;
        }
        const int norm = pairs[q].format == HH_PIX_U16;
        HH_K(HH_K_PREFILTER, 2, 0, 12.0 * P, P, hh::launch_u16_to_f32(a16, P, norm, dA, s));
        HH_K(HH_K_PREFILTER, 0, 0, 0, 0, hh::launch_u16_to_f32(b16, P, norm, dB, s));
        A = dA;
        B = dB;
      } else if (!device_inputs) {
        HH_CK(cudaMemcpyAsync(dA, A, P * sizeof(float), cudaMemcpyHostToDevice, s));
        HH_CK(cudaMemcpyAsync(dB, B, P * sizeof(float), cudaMemcpyHostToDevice, s));
        A = dA;
        B = dB;
      }
      if (k > 0) {
        HH_TRY(prefilter_pair(ctx, A, B, nr, nc, coefA, coefB));
        HH_K(HH_K_DEFORM, 1, 120.0 * P, 16.0 * P, P,
             hh::launch_deform(coefA, coefB, nr, nc, pred_src_u, pred_src_v, pg, warpA, warpB, s));
        A = warpA;
        B = warpB;
      }
      if (njobs > 0) {
        CorrArgs ca{};
        ca.A = A;
        ca.B = B;
        ca.mask = dmask;
        ca.ld = nr;
        ca.jobs = djobs;
        ca.njobs = njobs;
        ca.ny = ny;
        ca.G = G;
        ca.apod = tb.apod;
        ca.gain = tb.gain;
        ca.phasew = tb.phasew;
        ca.box_lo = tb.box_lo;
        ca.box_hi = tb.box_hi;
        ca.method = p.method;
        ca.npeaks = p.n_peaks;
        ca.finder = p.peak_finder;
        ca.subpixel = p.subpixel;
        ca.planes = acc;
        ca.accumulate = 1;
        ca.win = p.search[0] != W ? W : 0;
        ca.variant = corr_variant(ctx, p);
        if (!corr_special(p)) HH_TRY(gcorr_prepare(ctx, p, ca));
        HH_K(HH_K_CORRELATE, 1, corr_flops(p, njobs), corr_bytes(p, 0, njobs) + 8.0 * PL * njobs, njobs,
             corr_launch(ctx, p, ca, s));
        if (unc) {
          hh::UQArgs ua{};
          ua.A = A;
          ua.B = B;
          ua.mask = dmask;
          ua.ld = nr;
          ua.jobs = djobs;
          ua.njobs = njobs;
          ua.ny = ny;
          ua.W = W;
          ua.apod = tb.apod;
          ua.stats = stats;
          ua.accumulate = 1;
          HH_TRY(uq_prepare(ctx, p.window[0], p.window[1], ua));
          HH_K(HH_K_UQ, 1, uq_flops(p, njobs), 8.0 * p.window[0] * p.window[1] * njobs, njobs,
               hh::launch_uq(ua, s, ctx->num_sms));
        }
      }
    }
    // partial sums of this process's pairs -> sums over all processes
    if (ctx->ens_reduce && njobs > 0) {
      const int64_t nst = unc ? njobs * 88 : 0;
      if (ctx->ens_reduce(ctx->ens_reduce_user, k, acc, njobs * PL, unc ? stats : nullptr, nst, (void*)s) != 0)
        return fail(ctx, HH_ERR_STATE, "ensemble reducer failed in pass " + std::to_string(k + 1));
    }
    // ensemble_analyze! (src/ensemble.jl:273-305): one analysis of every summed plane
    if (unc && g.any_mask) {  // a masked cell has no estimate
      HH_K(HH_K_VECTOR, 1, 0, 4 * G, G, hh::launch_fill(uncu, NaN, G, s));
      HH_K(HH_K_VECTOR, 1, 0, 4 * G, G, hh::launch_fill(uncv, NaN, G, s));
    }
    if (njobs > 0) {
      hh::AnalyzeArgs aa{};
      aa.planes = acc;
      aa.nplanes = njobs;
      aa.nr = NR;
      aa.nc = NC;
      aa.npeaks = p.n_peaks;
      aa.finder = p.peak_finder;
      aa.subpixel = p.subpixel;
      aa.jobs = djobs;
      aa.ny = ny;
      aa.G = G;
      aa.du = resu;
      aa.dv = resv;
      aa.ratio = ratio;
      aa.moment = moment;
      aa.alt_u = nalt > 0 ? altu : nullptr;
      aa.alt_v = nalt > 0 ? altv : nullptr;
      aa.nalt = nalt;
      HH_K(HH_K_CORRELATE, 1, 0, 4.0 * PL * njobs, njobs, hh::launch_analyze_planes(aa, s));
      if (unc) HH_K(HH_K_UQ, 1, 0, 88.0 * 8 * njobs, njobs, hh::launch_uq_finalize(stats, djobs, njobs, ny, uncu, uncv, s));
    }
    HH_K(HH_K_VECTOR, 1, 0, (28 + 8 * nalt) * G, G,
         hh::launch_combine(u, v, resu, resv, ratio, moment, nalt > 0 ? altu : nullptr, nalt > 0 ? altv : nullptr, nalt,
                            g.any_mask ? gm : nullptr, ny, nx,
                            k > 0 ? node_pred(pred_src_u, pred_src_v, pg, g) : hh::NodePred{}, nullptr, nullptr, s));
    HH_TRY(validate_device(ctx, p, ny, nx, u, v, ratio, moment, outl, outl2, gm, g.any_mask,
                           nalt > 0 ? altu : nullptr, nalt > 0 ? altv : nullptr, nalt, force_replace));
    HH_CK(cudaEventRecord(ctx->events[k + 1], s));
  }
  if (out) HH_TRY(read_results(ctx, grids[np - 1], rb, Gmax, passes[np - 1].uncertainty != 0, out));
  else HH_CK(cudaStreamSynchronize(s));
  for (int k = 0; k < np; ++k) HH_CK(cudaEventElapsedTime(&ctx->pass_ms[k], ctx->events[k], ctx->events[k + 1]));
  return flush_profile(ctx);
}

extern "C" hh_status hh_set_ensemble_reducer(hh_ctx* ctx, hh_ensemble_reducer fn, void* user) {
  if (!ctx) return fail(nullptr, HH_ERR_ARG, "context is NULL");
  ctx->ens_reduce = fn;
  ctx->ens_reduce_user = fn ? user : nullptr;
  return HH_OK;
}
