// Multi-subject average with optional Fisher z (the reference's to_average
// modes, W/CorMat/CUCorMat/CUCorMat/CorMat.cpp:418-670) and the packed
// correlation matrix (.cormat) entry point.
#include "ctx.cuh"

// Every subject's z-scores (FP32 for the exact values, the form's operands
// for the tensor-core pass) and the subjects' two tables.  together: every
// subject's operands at once; else a subject's at a time (a split form's), its
// values added into sums / unc (unc may be null), which out then refers to: the
// memory of one subject's operands and N (N - 1) / 2 sums in the place of all
// operands, for studies whose operands do not fit beside the z-scores.
static int32_t avg_subjects(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                            const int32_t* T, int fisher, int prec, double delta_opt,
                            bool together, float* sums, uint32_t* unc, bna_ctx::Avg* out,
                            double* dsum, cudaStream_t st) {
  const int n_pad = round_up(N, kBlk), nb = n_pad / kBlk;
  const bool split = prec == BNA_PREC_BF16X3;
  if (!together && !split) return fail(ctx, BNA_OOM, "multi-subject call: out of device memory");
  size_t zn = 0, bn = 0;
  std::vector<size_t> zoff(nsub), boff(nsub);
  for (int k = 0; k < nsub; ++k) {
    zoff[k] = zn;
    boff[k] = together ? bn : 0;
    zn += (size_t)n_pad * round_up(T[k], 32);
    const size_t own = (size_t)n_pad * round_up(T[k], 64);
    bn = together ? bn + own : std::max(bn, own);
  }
  float* zall;
  uint8_t *badall, *bballs;
  void *subj_dev, *tc_dev, *vstat;
  uint16_t *zhi = nullptr, *zlo = nullptr;
  ENSURE(S_AVG_Z, zn * sizeof(float), zall);
  ENSURE(S_AVG_BAD, (size_t)nsub * n_pad, badall);
  ENSURE(S_BLOCKBAD, (size_t)nsub * nb, bballs);
  ENSURE(S_AVG_SUBJ, (size_t)nsub * avg_subj_bytes(), subj_dev);
  ENSURE(S_AVG_TC, (size_t)nsub * tc_subj_bytes(), tc_dev);
  ENSURE(S_VSTAT, zscore_scratch_bytes(n_pad), vstat);
  if (split) {
    ENSURE(S_AVG_ZHI, bn * 2, zhi);
    ENSURE(S_AVG_ZLO, bn * 2, zlo);
  }
  const int32_t s = tc_tiles(ctx, nb, st);
  if (s) return s;
  std::vector<char> subj_host((size_t)nsub * avg_subj_bytes());
  std::vector<char> tc_host((size_t)nsub * tc_subj_bytes());
  std::vector<CorrArgs> args(nsub);
  *dsum = 0;
  for (int k = 0; k < nsub; ++k) {
    CorrArgs& as = args[k];
    as.n = N;
    as.n_pad = n_pad;
    as.nb = nb;
    as.T = T[k];
    as.ldz = round_up(T[k], 32);
    as.ldb = round_up(T[k], 64);
    as.z = zall + zoff[k];
    as.zhi = split ? zhi + boff[k] : nullptr;
    as.zlo = split ? zlo + boff[k] : nullptr;
    as.bad = badall + (size_t)k * n_pad;
    const double dk = delta_opt > 0 ? delta_opt : default_delta(prec, T[k]);
    *dsum += dk;
    avg_subj_fill(subj_host.data(), k, as.z, as.bad, as.ldz, T[k]);
    if (!tc_subj_fill(tc_host.data(), k, as, bballs + (size_t)k * nb, split ? 0 : 1,
                      fisher ? 0.9f : (float)(1.0 - dk)))
      return fail(ctx, BNA_CUDA_ERROR, "multi-subject call: tensor map encoding failed");
  }
  CK(cudaMemcpyAsync(subj_dev, subj_host.data(), subj_host.size(), cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(tc_dev, tc_host.data(), tc_host.size(), cudaMemcpyHostToDevice, st));
  DevStatus* ds = nullptr;
  unsigned int* sched = nullptr;
  if (!together) {
    ENSURE(S_STATUS, sizeof(DevStatus), ds);
    CK(cudaMemsetAsync(ds, 0, sizeof(DevStatus), st));
    ENSURE(S_TCSCHED, 2 * sizeof(unsigned int), sched);
    CK(cudaMemsetAsync(sched, 0, 2 * sizeof(unsigned int), st));
  }
  for (int k = 0; k < nsub; ++k) {
    const CorrArgs& as = args[k];
    CK(launch_zscore(bold_dev[k], N, T[k], n_pad, const_cast<float*>(as.z), as.ldz,
                     const_cast<uint16_t*>(as.zhi), const_cast<uint16_t*>(as.zlo), as.ldb,
                     const_cast<uint8_t*>(as.bad), vstat, st, nullptr, 0, nullptr,
                     bballs + (size_t)k * nb));
    ctx->klaunch += 2;
    if (together) continue;
    CorrArgs a{};
    a.n = N;
    a.n_pad = n_pad;
    a.nb = nb;
    a.th.mode = BNA_THR_R_GE;
    a.th.tau = 2.0f;
    a.err = &ds->err;
    const AvgSums add{sums, unc, k > 0, true, nsub};
    const int2* tiles = reinterpret_cast<const int2*>(ctx->ptr[S_TILES]);
    const int per = ctx->tiles_per_launch > 0 ? ctx->tiles_per_launch : ctx->ntiles;
    for (int t0 = 0; t0 < ctx->ntiles; t0 += per, ++ctx->klaunch)
      CK(launch_corr_tc_avg(a, 4, split ? 0 : 1, static_cast<char*>(tc_dev) + k * tc_subj_bytes(),
                            1, fisher ? 1 : 0, tiles + t0, std::min(per, ctx->ntiles - t0), nullptr,
                            ctx->sms, sched, st, &add));
  }
  if (!together)
    CK(cudaMemcpyAsync(ctx->pinned, ds, sizeof(DevStatus), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));  // the host tables are released at return
  if (!together && (static_cast<const DevStatus*>(ctx->pinned)->err & ERR_TIMEOUT))
    return fail(ctx, BNA_TIMEOUT, "multi-subject sums: a bounded wait expired");
  *out = bna_ctx::Avg{subj_dev, tc_dev, nsub, fisher ? 1 : 0, AvgSums{}};
  if (!together) out->sums = AvgSums{sums, unc, true, false, nsub};
  return BNA_OK;
}

static int32_t avg_check(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                         const int32_t* T, int prec) {
  if (!ctx || nsub < 1 || !bold_dev || !T || N < 2)
    return fail(ctx, BNA_BAD_ARG, "multi-subject call: bad arguments");
  for (int k = 0; k < nsub; ++k)
    if (!bold_dev[k] || T[k] < 1)
      return fail(ctx, BNA_BAD_ARG, "subject %d: bad arguments", k);
  if (prec != BNA_PREC_BF16X3 && prec != BNA_PREC_TF32)
    return fail(ctx, BNA_UNSUPPORTED, "multi-subject call: a tensor-core form is required");
  return BNA_OK;
}

static int32_t csr_avg_once(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                            const int32_t* T, int32_t fisher, const bna_corr_opts* opts,
                            bna_csr* out_dev, bna_corr_stats* stats, void* stream,
                            bool together) {
  if (!opts || !out_dev || !T || nsub < 1)
    return fail(ctx, BNA_BAD_ARG, "bna_corr_csr_avg: bad arguments");
  int prec_r = opts->precision;
  int32_t s = resolve_precision(ctx, N, T[0], opts, &prec_r);
  if (s) return s;
  bna_corr_opts opts_r = *opts;
  opts_r.precision = prec_r;
  opts = &opts_r;
  s = avg_check(ctx, nsub, bold_dev, N, T, opts->precision);
  if (s) return s;
  if (!mode_known(opts->mode) ||
      (opts->mode == BNA_THR_DENSITY && !(opts->value >= 0.0 && opts->value <= 100.0)))
    return fail(ctx, BNA_BAD_ARG, "bna_corr_csr_avg: bad threshold rule");
  if (opts->mode == BNA_THR_R_EPS)
    return fail(ctx, BNA_UNSUPPORTED, "bna_corr_csr_avg: the 2mm tools' rule has no average");
  const int prec = opts->precision;
  s = set_device(ctx, as_stream(stream));
  if (s) return s;
  cudaStream_t st = as_stream(stream);
  ctx->klaunch = 0;
  ctx->last_ok = false;
  ctx->opt_used = true;  // the operands, or the sums
  const int n_pad = round_up(N, kBlk), nb = n_pad / kBlk;
  float* sums = nullptr;
  uint32_t* unc = nullptr;
  if (!together) {
    ENSURE(S_AVG_SUMS, (size_t)N * (N - 1) / 2 * sizeof(float), sums);
    ENSURE(S_AVG_UNC, avg_unc_words(nb) * sizeof(uint32_t), unc);
  }
  uint8_t* badz;
  ENSURE(S_AVG_BADZ, (size_t)n_pad, badz);
  CK(cudaMemsetAsync(badz, 0, (size_t)n_pad, st));
  CK(cudaEventRecord(ctx->ev[0], st));
  bna_ctx::Avg ac{};
  double dsum = 0;
  s = avg_subjects(ctx, nsub, bold_dev, N, T, fisher, prec, opts->delta, together, sums, unc, &ac,
                   &dsum, st);
  if (s) return s;
  CK(cudaEventRecord(ctx->ev[1], st));
  // bound of |average~ - average| (per-subject bounds, the float sums and
  // division; with Fisher z the transform's slope below |r| = 0.91, larger
  // |r~| being uncertain pairs that are always recomputed)
  const double dmean = dsum / nsub;
  const double u24 = std::ldexp(1.0, -24);
  const double davg = fisher ? 6.0 * dmean + 4e-6 + (nsub + 2) * 4.0 * u24
                             : dmean + (nsub + 1) * u24 + 4.0 * u24;
  CorrArgs a{};
  a.n = N;
  a.n_pad = n_pad;
  a.nb = nb;
  a.T = 1;
  a.ldz = 32;
  a.bad = badz;
  ctx->avg = &ac;
  s = corr_csr_core(ctx, a, N, 1, opts, prec, davg, out_dev, stats, st);
  ctx->avg = nullptr;
  return s;
}

// once(together); where memory does not reach, again without what earlier calls
// left of the optional workspaces, then with one subject's operands at a time (the
// split form's: the other has none beside the z-scores).
template <class F>
static int32_t avg_tries(bna_ctx* ctx, int32_t nsub, F once) {
  int32_t s = once(true);
  for (int k = 0; s == BNA_OOM && k < (nsub > 1 ? 2 : 1); ++k) {
    release_optional(ctx);
    s = once(k == 0);
  }
  return s;
}

int32_t bna_corr_csr_avg(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                         const int32_t* T, int32_t fisher, const bna_corr_opts* opts,
                         bna_csr* out_dev, bna_corr_stats* stats, void* stream) {
  return avg_tries(ctx, nsub, [&](bool together) {
    return csr_avg_once(ctx, nsub, bold_dev, N, T, fisher, opts, out_dev, stats, stream, together);
  });
}

static int32_t packed_once(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                           const int32_t* T, int32_t fisher, int32_t precision, float* packed_dev,
                           void* stream, bool together) {
  int32_t s = avg_check(ctx, nsub, bold_dev, N, T, precision);
  if (s) return s;
  if (!packed_dev) return fail(ctx, BNA_BAD_ARG, "bna_corr_packed: packed_dev is NULL");
  s = set_device(ctx, as_stream(stream));
  if (s) return s;
  cudaStream_t st = as_stream(stream);
  ctx->klaunch = 0;
  ctx->last_ok = false;
  ctx->opt_used = true;
  bna_ctx::Avg ac{};
  double dsum = 0;
  // (the caller's matrix serves for the sums)
  s = avg_subjects(ctx, nsub, bold_dev, N, T, fisher, precision, 0.0, together, packed_dev, nullptr,
                   &ac, &dsum, st);
  if (s) return s;
  CorrArgs a{};
  a.n = N;
  a.n_pad = round_up(N, kBlk);
  a.nb = a.n_pad / kBlk;
  a.th.mode = BNA_THR_R_GE;
  a.th.tau = 2.0f;
  DevStatus* ds;
  ENSURE(S_STATUS, sizeof(DevStatus), ds);
  CK(cudaMemsetAsync(ds, 0, sizeof(DevStatus), st));
  a.err = &ds->err;
  const int2* tiles = reinterpret_cast<const int2*>(ctx->ptr[S_TILES]);
  const int per = ctx->tiles_per_launch > 0 ? ctx->tiles_per_launch : ctx->ntiles;
  unsigned int* sched;
  ENSURE(S_TCSCHED, 2 * sizeof(unsigned int), sched);
  CK(cudaMemsetAsync(sched, 0, 2 * sizeof(unsigned int), st));
  for (int t0 = 0; t0 < ctx->ntiles; t0 += per, ++ctx->klaunch)
    CK(launch_corr_tc_avg(a, 4, precision == BNA_PREC_BF16X3 ? 0 : 1, ac.tc,
                          together ? nsub : 0, ac.fisher, tiles + t0,
                          std::min(per, ctx->ntiles - t0), packed_dev, ctx->sms, sched, st,
                          together ? nullptr : &ac.sums));
  DevStatus* hs = reinterpret_cast<DevStatus*>(ctx->pinned);
  CK(cudaMemcpyAsync(hs, ds, sizeof(DevStatus), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (hs->err & ERR_TIMEOUT) return fail(ctx, BNA_TIMEOUT, "packed matrix: a bounded wait expired");
  return BNA_OK;
}

int32_t bna_corr_packed(bna_ctx* ctx, int32_t nsub, const float* const* bold_dev, int32_t N,
                        const int32_t* T, int32_t fisher, int32_t precision, float* packed_dev,
                        void* stream) {
  return avg_tries(ctx, nsub, [&](bool together) {
    return packed_once(ctx, nsub, bold_dev, N, T, fisher, precision, packed_dev, stream, together);
  });
}
