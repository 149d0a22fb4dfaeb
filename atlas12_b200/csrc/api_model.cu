// api_model.cu -- device-resident ATLAS12 model: the iteration loop of
// atlas12c.f90:496-606 with every step on the device, one CUDA graph per
// iteration.  The EOS / populations / continuum come from the synthetic
// surrogate (surrogate.cuh) that stands in for the off-path physics.
#include <cmath>
#include <vector>

#include "api_common.cuh"
#include "model.cuh"

using namespace atlasgpu;

struct atlasgpu_model {
  int nrhox, kw, numnu, nwave, nspec;
  int64_t nlines;
  double teff, grav, vturb, mh;
  // device memory
  double* state;         // [kNState][kw]
  ModelState* ms;        // device struct pointing into state
  double *xnfdop, *dopple;  // [nspec][kw]
  double *xne_eos, *txnxn, *hkt, *hckt, *rho;  // [kw]
  ContCoef* cc;          // [kw]
  double *acont, *sigmac;  // the RT pass's continuum [numnu][kw]
  double *waveset, *rcoset, *cutwave, *tabcont;  // tabcont [nwave+1][kw]
  int32_t* iwavetab;
  int32_t* linedata;
  AtlasLine* lines;
  double* xl;            // XLINES(J, NU): [numnu][kw]
  unsigned long long* xfix;  // LINOP1's exact fixed-point sums [numnu][3][kw]
  int* fscale;             // the exponents k of their per-depth scales 2^k [kw]
  double* funscale;        // 2^-k [kw]
  unsigned long long* cgfmax;  // largest CGF per species [nspec] (FP64 bit patterns)
  double *partial, *sum, *hsurf;
  double *h0, *h1, *h2, *ross;  // ross: ROSSTAB points [3][kRossMax]
  float4* hf;                    // FP32 (H0, H1, H2, 0)
  RossStore* R;                  // device
  int* iter_dev;         // iterations completed
  double* maxerr_dev;    // last max |FLXERR|
  unsigned long long* cnt;
  int nwl;                 // partial-sum rows allocated
  RtSplitShape rt_sh;      // launch shape of the split RT pass over the shard
  double* rt_rec;          // the split pass's per-frequency records [rt_rec_doubles(numnu, kw)]
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  int graph_precision = -1;  // precision the captured graph was built with
  int nu_first = 1, nu_last = 0;  // frequency shard (1-based, inclusive; 0 = NUMNU)
  double* ext_sums = nullptr;     // caller-owned device buffer for the frequency sums (or null)
  bool kapcont_done = false;
};

namespace {

// hydrostatics (iteration > 1), surrogate EOS / populations, Planck factors
__global__ void k_model_eos(ModelState* ms, const int* iter_dev, int nrhox, int kw, double grav,
                            double vturb_cms, double mh, double* xnfdop, double* dopple, double* xne_eos,
                            double* txnxn, double* hkt, double* hckt, double* rho, ContCoef* cc, int nspec,
                            const double* cgfmax, int* fscale, double* funscale) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (j >= nrhox) return;
  model_eos_depth(lane, ms, *iter_dev + 1, j, kw, grav, vturb_cms, mh, xnfdop, dopple, xne_eos, txnxn, hkt, hckt, rho,
                  cc);
  __syncwarp();
  fix_scale_depth(lane, xnfdop, nspec, kw, j, cgfmax, fscale, funscale);
}

// KAPCONT (atlas12_modules.f90:19072-19138) on the surrogate continuum
__global__ void k_model_kapcont(const double* cutwave, int nwave, const double* waveset, int nrhox,
                                int kw, const double* hkt, const ContCoef* cc, double* tabcont) {
  model_kapcont_row(blockIdx.x, cutwave, nwave, waveset, nrhox, kw, hkt, cc, tabcont);
}

__global__ void __launch_bounds__(kFinThreads) k_model_finish(ModelState* ms, double* acc, int kw, int n,
                                                               int* iter_dev, double teff, double grav,
                                                               RossStore* R, double* maxerr) {
  extern __shared__ __align__(16) double fin_smem[];
  if (blockIdx.x != 0) return;
  const int iter = *iter_dev + 1;
  __syncthreads();  // every thread has read the count before thread 0 advances it
  const double e = b_atlas_finish(ms, acc, kw, n, iter, teff, grav, R, fin_smem);
  if (threadIdx.x == 0) {
    *maxerr = e;
    *iter_dev = iter;
  }
}

// KAPP stand-in for the RT pass: ACONT, SIGMAC [numnu][kw]
__global__ void k_model_kapp(const double* waveset, int numnu, int nrhox, int kw, const ContCoef* cc,
                             double* acont, double* sigmac) {
  model_kapp_range(waveset, numnu, nrhox, kw, cc, acont, sigmac, nullptr);
}

__global__ void k_surrogate_eval(int nrhox, const double* t, const double* p, double vturb_cms, int nw,
                                 const double* wave, double* xnfdop, double* dopple, ContCoef* cc,
                                 double* kabs, double* sigma, double* xne, double* rho) {
  const int j = blockIdx.x;
  if (j >= nrhox) return;
  if (threadIdx.x < 32) {
    const EosOut e = surrogate_depth(threadIdx.x, t[j], p[j], vturb_cms, 0.0, j, nrhox, xnfdop, dopple, cc + j);
    if (threadIdx.x == 0) {
      xne[j] = e.xne;
      rho[j] = e.rho;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nw; i += blockDim.x) {
    double ka, sg;
    surrogate_kapp(cc[j], wave[i], ka, sg);
    kabs[(size_t)i * nrhox + j] = ka;
    sigma[(size_t)i * nrhox + j] = sg;
  }
}

// RT launch shape for the model's frequency shard: enough warps and pair
// groups to fill every SM several times, frequencies contiguous per unit
void rt_shape(atlasgpu_ctx* ctx, atlasgpu_model* m) {
  const int last = m->nu_last > 0 ? m->nu_last : m->numnu;
  m->rt_sh = rt_split_shape(last - m->nu_first + 1, ctx->nsm, 1, 4);
}

// The first part of one iteration on the context stream, up to the reduced
// frequency sums (EOS, KAPCONT on the first iteration, LINOP1, KAPP, the RT
// pass over the model's shard, the fixed-order reduction).  With timed =
// true (never while a graph is being captured) each launch is bracketed by
// CUDA events.
int enqueue_begin(atlasgpu_ctx* ctx, atlasgpu_model* m, bool timed) {
  cudaStream_t s = ctx->stream;
  const bool was = ctx->timing;
  ctx->timing = was && timed;
  {
    Timer tm(ctx, "model_eos");
    k_model_eos<<<(m->nrhox + 3) / 4, 128, 0, s>>>(m->ms, m->iter_dev, m->nrhox, m->kw, m->grav, m->vturb * 1.0e5, m->mh,
                                  m->xnfdop,
                                  m->dopple, m->xne_eos, m->txnxn, m->hkt, m->hckt, m->rho, m->cc, m->nspec,
                                  (const double*)m->cgfmax, m->fscale, m->funscale);
    CKL(ctx);
  }
  if (!m->kapcont_done) {
    k_model_kapcont<<<m->nwave, 128, 0, s>>>(m->cutwave, m->nwave, m->waveset, m->nrhox, m->kw, m->hkt,
                                             m->cc, m->tabcont);
    CKL(ctx);
  }
  if (m->nlines == 0) CK(cudaMemsetAsync(m->xl, 0, (size_t)m->kw * m->numnu * sizeof(double), s));
  if (m->nlines > 0) {
    LinopArgs la{m->lines, m->nlines, m->nrhox, m->kw, m->nspec, m->numnu, m->xnfdop, m->dopple,
                 m->xne_eos, m->txnxn, m->hckt, m->tabcont, m->waveset, m->h0, m->h1, m->h2, m->hf, m->xl,
                 nullptr, m->cnt, m->nu_first, m->nu_last};
    la.work = work_counters(ctx, 1);
    la.xfix = m->xfix;
    la.fscale = m->fscale;
    {
      Timer tm(ctx, "atlas_linop");
      linop_launch(ctx, la);
      CKL(ctx);
      k_fix_finalize<<<grid_for(ctx, (int64_t)m->numnu * m->nrhox, 256, 8), 256, 0, s>>>(
          m->xfix, m->funscale, m->numnu, m->nrhox, m->kw, m->xl);
      CKL(ctx);
    }
    work_collect(ctx, la.work, {"atlas_linop_points"});
  }
  {
    Timer tm(ctx, "model_kapp");
    k_model_kapp<<<grid_for(ctx, (int64_t)m->numnu * m->nrhox, 256, 8), 256, 0, s>>>(
        m->waveset, m->numnu, m->nrhox, m->kw, m->cc, m->acont, m->sigmac);
    CKL(ctx);
  }
  RtArgs ra{ctx->ops, m->numnu, m->nrhox, m->kw, m->waveset, m->rcoset, m->acont, m->sigmac, nullptr,
            m->xl, (const double*)m->state + 1 * m->kw, (const double*)m->state + 0 * m->kw, m->hkt,
            m->teff, 1, 1, m->kw, m->partial, m->hsurf, nullptr, m->nu_first, m->nu_last};
  const RtSplitShape& sh = m->rt_sh;
  rt_split_args(ra, sh);
  ra.rec = m->rt_rec;
  double* sums = m->ext_sums ? m->ext_sums : m->sum;
  {
    Timer tm(ctx, "atlas_rt");
    k_rt_pre<<<sh.pre_blocks, kRtSplitWarps * 32, rt_pre_smem_bytes(), s>>>(ra);
    CKL(ctx);
    k_rt_series<<<sh.series_blocks, kScatterThreads, 0, s>>>(ra);
    CKL(ctx);
    k_rt_solve<<<sh.solve_blocks, kScatterThreads, scatter_smem_bytes(), s>>>(ra);
    CKL(ctx);
    k_rt_post<<<sh.post_blocks, kRtSplitWarps * 32, rt_post_smem_bytes(m->nrhox), s>>>(ra);
    CKL(ctx);
  }
  {
    Timer tm(ctx, "atlas_reduce");
    launch_reduce(m->partial, sh.rows(), m->kw, sums, s);
    CKL(ctx);
  }
  ctx->timing = was;
  return 0;
}

// The rest of the iteration: ROSS(3), RADIAP(3), TCORR(3) and the remap from
// the (possibly externally all-reduced) frequency sums.
int enqueue_finish(atlasgpu_ctx* ctx, atlasgpu_model* m, bool timed) {
  cudaStream_t s = ctx->stream;
  const bool was = ctx->timing;
  ctx->timing = was && timed;
  double* sums = m->ext_sums ? m->ext_sums : m->sum;
  {
    Timer tm(ctx, "atlas_finish");
    k_model_finish<<<1, kFinThreads, fin_smem_bytes(m->kw, kRossMax), s>>>(
        m->ms, sums, m->kw, m->nrhox, m->iter_dev, m->teff, m->grav, m->R, m->maxerr_dev);
    CKL(ctx);
  }
  ctx->timing = was;
  return 0;
}

int enqueue_iteration(atlasgpu_ctx* ctx, atlasgpu_model* m, bool timed) {
  int r;
  if ((r = enqueue_begin(ctx, m, timed))) return r;
  return enqueue_finish(ctx, m, timed);
}

void drop_graph(atlasgpu_model* m) {
  if (m->gexec) cudaGraphExecDestroy(m->gexec);
  if (m->graph) cudaGraphDestroy(m->graph);
  m->gexec = nullptr;
  m->graph = nullptr;
}

__global__ void k_fp64_fma(double* out, int iters) {
  // 8 independent DFMA chains per thread
  double a[8];
  for (int k = 0; k < 8; ++k) a[k] = 1.0 + 1e-9 * (threadIdx.x + k);
  const double b = 0.999999999, c = 1e-12;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
  }
  double s = 0.0;
  for (int k = 0; k < 8; ++k) s += a[k];
  if (s == 12345.678) out[0] = s;  // keep the chains alive
}

// 64-bit integer atomic adds at L2, lanes of a warp on 32 consecutive words
// (as LINOP1's lanes at consecutive depths), warps scattered over the region
__global__ void k_u64_atomics(unsigned long long* w, size_t nwords, int iters) {
  const size_t warp = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const size_t nrows = nwords / 32;
  for (int i = 0; i < iters; ++i) {
    const size_t row = (warp * 7919u + (size_t)i * 104729u) % nrows;
    atomicAdd(w + row * 32 + lane, 1ull);
  }
}

template <class T>
int dalloc(atlasgpu_ctx* ctx, T** p, size_t n) {
  if (cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, ATLASGPU_ENOMEM, "model: cudaMalloc of %zu bytes", n * sizeof(T));
  }
  return 0;
}

}  // namespace

extern "C" {

int atlasgpu_surrogate_eval(atlasgpu_ctx* ctx, int nrhox, const double* t, const double* p, double vturb_kms,
                            int nw, const double* wave, double* kabs, double* sigma, double* xne,
                            double* xnfdop) {
  if (!ctx || nrhox < 1 || nrhox > kKwMax || nw < 1 || !t || !p || !wave || !kabs || !sigma || !xne)
    return fail(ctx, ATLASGPU_EINVAL, "surrogate_eval: bad argument");
  cudaSetDevice(ctx->device);
  double *dt, *dp, *dw, *dxd, *ddp, *dka, *dsg, *dxne, *drho;
  ContCoef* dcc;
  int r;
  const size_t ns = (size_t)kSurrNspec * nrhox;
  if ((r = bufT(ctx, "se_t", nrhox, &dt)) || (r = bufT(ctx, "se_p", nrhox, &dp)) || (r = bufT(ctx, "se_w", nw, &dw)) ||
      (r = bufT(ctx, "se_xd", ns, &dxd)) || (r = bufT(ctx, "se_dp", ns, &ddp)) ||
      (r = bufT(ctx, "se_ka", (size_t)nw * nrhox, &dka)) || (r = bufT(ctx, "se_sg", (size_t)nw * nrhox, &dsg)) ||
      (r = bufT(ctx, "se_xne", nrhox, &dxne)) || (r = bufT(ctx, "se_rho", nrhox, &drho)) ||
      (r = bufT(ctx, "se_cc", nrhox, &dcc)))
    return r;
  cudaStream_t s = ctx->stream;
  CK(cudaMemcpyAsync(dt, t, nrhox * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(dp, p, nrhox * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(dw, wave, nw * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemsetAsync(dxd, 0, ns * sizeof(double), s));
  k_surrogate_eval<<<nrhox, 128, 0, s>>>(nrhox, dt, dp, vturb_kms * 1.0e5, nw, dw, dxd, ddp, dcc, dka, dsg, dxne, drho);
  CKL(ctx);
  CK(cudaMemcpyAsync(kabs, dka, (size_t)nw * nrhox * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(sigma, dsg, (size_t)nw * nrhox * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(xne, dxne, nrhox * sizeof(double), cudaMemcpyDeviceToHost, s));
  if (xnfdop) CK(cudaMemcpyAsync(xnfdop, dxd, ns * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return 0;
}

int atlasgpu_model_create(atlasgpu_ctx* ctx, const atlasgpu_model_desc* d, atlasgpu_model** out) {
  if (!ctx || !d || !out) return fail(ctx, ATLASGPU_EINVAL, "model_create: null argument");
  *out = nullptr;
  if (!ctx->ops_set) return fail(ctx, ATLASGPU_ESTATE, "model_create: operators not set");
  if (d->nrhox < 16 || d->nrhox > kKwMax || d->numnu < 2 || d->nwave < 1 || d->nlines < 0 || !d->t || !d->p ||
      !d->rhox || !d->tauros || !d->waveset || !d->rcoset || !d->cutoff_wave || (d->nlines > 0 && !d->linedata) ||
      !d->h0tab || !d->h1tab || !d->h2tab || !(d->teff > 0) || !(d->vturb_kms >= 0))
    return fail(ctx, ATLASGPU_EINVAL, "model_create: bad descriptor");
  for (int i = 1; i < d->numnu; ++i)
    if (!(d->waveset[i] > d->waveset[i - 1])) return fail(ctx, ATLASGPU_EINVAL, "WAVESET not increasing");
  for (int i = 1; i < d->nwave; ++i)
    if (!(d->cutoff_wave[i] > d->cutoff_wave[i - 1])) return fail(ctx, ATLASGPU_EINVAL, "cutoff grid not increasing");
  cudaSetDevice(ctx->device);
  atlasgpu_model* m = new atlasgpu_model();
  m->nrhox = d->nrhox;
  m->kw = d->nrhox;
  m->numnu = d->numnu;
  m->nwave = d->nwave;
  m->nspec = kSurrNspec;
  m->nlines = d->nlines;
  m->teff = d->teff;
  m->grav = pow(10.0, d->logg);
  m->vturb = d->vturb_kms;
  m->mh = d->mh;
  const int kw = m->kw;
  int r = 0;
  const size_t nr = (size_t)3 * kRossMax;
  if ((r = dalloc(ctx, &m->state, kNState * kw)) || (r = dalloc(ctx, &m->ms, 1)) ||
      (r = dalloc(ctx, &m->xnfdop, (size_t)m->nspec * kw)) || (r = dalloc(ctx, &m->dopple, (size_t)m->nspec * kw)) ||
      (r = dalloc(ctx, &m->xne_eos, kw)) || (r = dalloc(ctx, &m->txnxn, kw)) || (r = dalloc(ctx, &m->hkt, kw)) ||
      (r = dalloc(ctx, &m->hckt, kw)) || (r = dalloc(ctx, &m->rho, kw)) || (r = dalloc(ctx, &m->cc, kw)) ||
      (r = dalloc(ctx, &m->acont, (size_t)m->numnu * kw)) || (r = dalloc(ctx, &m->sigmac, (size_t)m->numnu * kw)) ||
      (r = dalloc(ctx, &m->waveset, m->numnu)) || (r = dalloc(ctx, &m->rcoset, m->numnu)) ||
      (r = dalloc(ctx, &m->cutwave, m->nwave)) || (r = dalloc(ctx, &m->tabcont, (size_t)(m->nwave + 1) * kw)) ||
      (r = dalloc(ctx, &m->iwavetab, m->nwave + 1)) || (r = dalloc(ctx, &m->linedata, (size_t)m->nlines * 4)) ||
      (r = dalloc(ctx, &m->lines, (size_t)m->nlines)) || (r = dalloc(ctx, &m->xl, (size_t)kw * m->numnu)) ||
      (r = dalloc(ctx, &m->xfix, (size_t)kFixWords * kw * m->numnu)) || (r = dalloc(ctx, &m->fscale, kw)) ||
      (r = dalloc(ctx, &m->funscale, kw)) || (r = dalloc(ctx, &m->cgfmax, (size_t)m->nspec)) ||
      (r = dalloc(ctx, &m->sum, kAcc * kw + 1)) ||
      (r = dalloc(ctx, &m->hsurf, m->numnu)) || (r = dalloc(ctx, &m->h0, 2001)) || (r = dalloc(ctx, &m->h1, 2001)) ||
      (r = dalloc(ctx, &m->h2, 2001)) || (r = dalloc(ctx, &m->hf, 2001)) || (r = dalloc(ctx, &m->ross, nr)) || (r = dalloc(ctx, &m->R, 1)) || (r = dalloc(ctx, &m->iter_dev, 1)) ||
      (r = dalloc(ctx, &m->maxerr_dev, 1)) || (r = dalloc(ctx, &m->cnt, 2))) {
    atlasgpu_model_destroy(ctx, m);
    return r;
  }
  // RT launch shape, partial sums for the most rows any shard can need, records
  rt_shape(ctx, m);
  m->nwl = rt_split_rows_max(m->numnu, ctx->nsm, 4);
  if ((r = dalloc(ctx, &m->partial, (size_t)m->nwl * (kAcc * kw + 1))) ||
      (r = dalloc(ctx, &m->rt_rec, rt_rec_doubles(m->numnu, kw)))) {
    atlasgpu_model_destroy(ctx, m);
    return r;
  }
  CK(rt_split_attributes(m->nrhox));
  if (fin_smem_bytes(kw, kRossMax) > (size_t)ctx->smem_optin) {
    atlasgpu_model_destroy(ctx, m);
    return fail(ctx, ATLASGPU_EINVAL, "model_create: finish needs %zu B of shared memory",
                fin_smem_bytes(kw, kRossMax));
  }
  CK(cudaFuncSetAttribute(k_model_finish, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)fin_smem_bytes(kw, kRossMax)));
  cudaStream_t s = ctx->stream;
  // state vectors: t, rhox, p, xne, abross, prad, vturb, pturb, tauros, accrad, raden, oldt1, flxerr,
  // dtflux, dtlamb, dtsurf, t1
  std::vector<double> h(kNState * kw, 0.0);
  for (int j = 0; j < kw; ++j) {
    h[0 * kw + j] = d->t[j];
    h[1 * kw + j] = d->rhox[j];
    h[2 * kw + j] = d->p[j];
    h[6 * kw + j] = d->vturb_kms * 1.0e5;
    h[8 * kw + j] = d->tauros[j];
  }
  ModelState ms;
  double** f[kNState] = {&ms.t, &ms.rhox, &ms.p, &ms.xne, &ms.abross, &ms.prad, &ms.vturb, &ms.pturb, &ms.tauros,
                         &ms.accrad, &ms.raden, &ms.oldt1, &ms.flxerr, &ms.dtflux, &ms.dtlamb, &ms.dtsurf, &ms.t1};
  for (int q = 0; q < kNState; ++q) *f[q] = m->state + q * kw;
  ms.pradk0 = 0.0;
  ms.maxerr = 0.0;
  CK(cudaMemcpyAsync(m->state, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->ms, &ms, sizeof ms, cudaMemcpyHostToDevice, s));
  CK(cudaMemsetAsync(m->xnfdop, 0, (size_t)m->nspec * kw * sizeof(double), s));
  // dopple must be nonzero where a line may look: fill with 1 (the populations are 0 there)
  {
    std::vector<double> one((size_t)m->nspec * kw, 1.0);
    CK(cudaMemcpy(m->dopple, one.data(), one.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  CK(cudaMemcpyAsync(m->waveset, d->waveset, m->numnu * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->rcoset, d->rcoset, m->numnu * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->cutwave, d->cutoff_wave, m->nwave * sizeof(double), cudaMemcpyHostToDevice, s));
  std::vector<int32_t> iwt(m->nwave + 1);
  const double RATIOLG = log(1.0 + 1.0 / 2000000.0);
  for (int i = 0; i < m->nwave; ++i) iwt[i] = (int32_t)(log(d->cutoff_wave[i]) / RATIOLG + 0.5);
  iwt[m->nwave] = 1 << 30;
  CK(cudaMemcpyAsync(m->iwavetab, iwt.data(), iwt.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  if (m->nlines > 0)
    CK(cudaMemcpyAsync(m->linedata, d->linedata, (size_t)m->nlines * 4 * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->h0, d->h0tab, 2001 * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->h1, d->h1tab, 2001 * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(m->h2, d->h2tab, 2001 * sizeof(double), cudaMemcpyHostToDevice, s));
  {
    const std::vector<float4> hf = pack_voigt_f32(d->h0tab, d->h1tab, d->h2tab, 2001);
    CK(cudaMemcpy(m->hf, hf.data(), hf.size() * sizeof(float4), cudaMemcpyHostToDevice));
  }
  {
    RossStore R0{0, kRossMax, 0.0, 1.0, 0.0, 1.0, m->ross, m->ross + kRossMax, m->ross + 2 * kRossMax};
    CK(cudaMemcpy(m->R, &R0, sizeof R0, cudaMemcpyHostToDevice));
  }
  CK(cudaMemsetAsync(m->iter_dev, 0, sizeof(int), s));
  CK(cudaMemsetAsync(m->cnt, 0, 2 * sizeof(unsigned long long), s));
  // TABLOG and the per-line preparation (iteration invariant)
  double* tl;
  {
    const bool fresh = ctx->bufs.find("tablog") == ctx->bufs.end();
    if ((r = bufT(ctx, "tablog", 65536, &tl))) {
      atlasgpu_model_destroy(ctx, m);
      return r;
    }
    if (fresh) {
      std::vector<double> ht(65536);
      for (int k = 0; k < 65536; ++k) ht[k] = pow(10.0, (double)((k - 32768) - 16384) * 0.001);
      CK(cudaMemcpy(tl, ht.data(), 65536 * sizeof(double), cudaMemcpyHostToDevice));
    }
  }
  if (m->nlines > 0 && (r = atlas_prep_lines(ctx, m->linedata, d->linedata, m->nlines, tl, m->waveset, d->waveset,
                                              m->numnu, m->iwavetab, m->nwave, m->nspec, m->lines))) {
    atlasgpu_model_destroy(ctx, m);
    return r;
  }
  // exact XLINES sums: zeroed words, the largest CGF per species for the scales
  CK(cudaMemsetAsync(m->xfix, 0, (size_t)kFixWords * kw * m->numnu * sizeof(unsigned long long), s));
  CK(cudaMemsetAsync(m->cgfmax, 0, (size_t)m->nspec * sizeof(unsigned long long), s));
  if (m->nlines > 0) {
    k_cgf_max<<<grid_for(ctx, m->nlines, 256, 8), 256, 0, s>>>(m->lines, m->nlines, m->nspec, m->cgfmax);
    CKL(ctx);
  }
  CK(cudaStreamSynchronize(s));
  *out = m;
  return 0;
}

int atlasgpu_model_iterate(atlasgpu_ctx* ctx, atlasgpu_model* m, int max_iter, double tol, int use_graph,
                           int* iters_done, double* hist) {
  if (!ctx || !m || max_iter < 0) return fail(ctx, ATLASGPU_EINVAL, "model_iterate: bad argument");
  cudaSetDevice(ctx->device);
  cudaStream_t s = ctx->stream;
  int done = 0, r;
  Timer tm(ctx, "model_iterate");
  for (int it = 0; it < max_iter; ++it) {
    if (!m->kapcont_done) {
      // first iteration of the model: KAPCONT included, not captured
      if ((r = enqueue_iteration(ctx, m, true))) return r;
      m->kapcont_done = true;
    } else if (use_graph) {
      if (m->gexec && m->graph_precision != ctx->precision) {
        cudaGraphExecDestroy(m->gexec);
        cudaGraphDestroy(m->graph);
        m->gexec = nullptr;
        m->graph = nullptr;
      }
      if (!m->gexec) {
        CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const int64_t l0 = ctx->launches;
        r = enqueue_iteration(ctx, m, false);
        cudaGraph_t g = nullptr;
        const cudaError_t ec = cudaStreamEndCapture(s, &g);
        if (r) return r;
        if (ec != cudaSuccess) return fail(ctx, ATLASGPU_ECUDA, "graph capture: %s", cudaGetErrorString(ec));
        m->graph = g;
        CK(cudaGraphInstantiate(&m->gexec, g, 0));
        m->graph_precision = ctx->precision;
        ctx->launches = l0;  // counted when replayed
      }
      CK(cudaGraphLaunch(m->gexec, s));
      ctx->launches += m->nlines > 0 ? 7 : 5;
    } else {
      if ((r = enqueue_iteration(ctx, m, true))) return r;
    }
    double e = 0.0;
    CK(cudaMemcpyAsync(&e, m->maxerr_dev, sizeof e, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (hist) hist[it] = e;
    ++done;
    if (!(e == e)) return fail(ctx, ATLASGPU_ENONFINITE, "model_iterate: FLXERR is not finite at iteration %d", done);
    if (tol > 0.0 && e <= tol) break;
  }
  tm.stop();
  if (iters_done) *iters_done = done;
  return 0;
}

int atlasgpu_model_get(atlasgpu_ctx* ctx, atlasgpu_model* m, double* t, double* rhox, double* p, double* xne,
                       double* flxerr, double* hsurf) {
  if (!ctx || !m) return fail(ctx, ATLASGPU_EINVAL, "model_get: null");
  cudaSetDevice(ctx->device);
  const int kw = m->kw;
  std::vector<double> h(kNState * kw);
  CK(cudaMemcpyAsync(h.data(), m->state, h.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if (hsurf) CK(cudaMemcpyAsync(hsurf, m->hsurf, m->numnu * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  if (t) memcpy(t, h.data() + 0 * kw, m->nrhox * sizeof(double));
  if (rhox) memcpy(rhox, h.data() + 1 * kw, m->nrhox * sizeof(double));
  if (p) memcpy(p, h.data() + 2 * kw, m->nrhox * sizeof(double));
  if (xne) memcpy(xne, h.data() + 3 * kw, m->nrhox * sizeof(double));
  if (flxerr) memcpy(flxerr, h.data() + 12 * kw, m->nrhox * sizeof(double));
  return 0;
}

int atlasgpu_model_get_tables(atlasgpu_ctx* ctx, atlasgpu_model* m, double* tabcont, double* xlines, double* acont,
                              double* sigmac) {
  if (!ctx || !m) return fail(ctx, ATLASGPU_EINVAL, "model_get_tables: null");
  cudaSetDevice(ctx->device);
  cudaStream_t s = ctx->stream;
  const size_t nn = (size_t)m->numnu * m->kw * sizeof(double);
  if (tabcont)
    CK(cudaMemcpyAsync(tabcont, m->tabcont, (size_t)(m->nwave + 1) * m->kw * sizeof(double), cudaMemcpyDeviceToHost,
                       s));
  if (xlines) CK(cudaMemcpyAsync(xlines, m->xl, nn, cudaMemcpyDeviceToHost, s));
  if (acont) CK(cudaMemcpyAsync(acont, m->acont, nn, cudaMemcpyDeviceToHost, s));
  if (sigmac) CK(cudaMemcpyAsync(sigmac, m->sigmac, nn, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return 0;
}

int atlasgpu_model_set_structure(atlasgpu_ctx* ctx, atlasgpu_model* m, const double* t, const double* p,
                                 const double* rhox) {
  if (!ctx || !m || !t || !p || !rhox) return fail(ctx, ATLASGPU_EINVAL, "model_set_structure: null");
  cudaSetDevice(ctx->device);
  const int kw = m->kw;
  CK(cudaStreamSynchronize(ctx->stream));
  // a fresh model, as atlasgpu_model_create leaves it: every state vector
  // zero except T, RHOX, P, VTURB (kept) and TAUROS = TAUSTD, so nothing of
  // the previous model (or of a failed, non-finite one) carries over
  std::vector<double> h(kNState * kw);
  CK(cudaMemcpy(h.data(), m->state, h.size() * sizeof(double), cudaMemcpyDeviceToHost));
  for (int q = 0; q < kNState; ++q)
    if (q != 6)
      for (int j = 0; j < kw; ++j) h[q * kw + j] = 0.0;
  for (int j = 0; j < m->nrhox; ++j) {
    h[0 * kw + j] = t[j];
    h[1 * kw + j] = rhox[j];
    h[2 * kw + j] = p[j];
    h[8 * kw + j] = pow(10.0, -6.875 + 0.125 * j);
  }
  CK(cudaMemcpy(m->state, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
  {
    ModelState ms;
    CK(cudaMemcpy(&ms, m->ms, sizeof ms, cudaMemcpyDeviceToHost));
    ms.pradk0 = 0.0;
    ms.maxerr = 0.0;
    CK(cudaMemcpy(m->ms, &ms, sizeof ms, cudaMemcpyHostToDevice));
  }
  CK(cudaMemset(m->iter_dev, 0, sizeof(int)));
  m->kapcont_done = false;  // KAPCONT runs again on the new structure's first iteration
  RossStore R0{0, kRossMax, 0.0, 1.0, 0.0, 1.0, m->ross, m->ross + kRossMax, m->ross + 2 * kRossMax};
  CK(cudaMemcpy(m->R, &R0, sizeof R0, cudaMemcpyHostToDevice));
  return 0;
}

int atlasgpu_model_set_params(atlasgpu_ctx* ctx, atlasgpu_model* m, double teff, double logg,
                              double vturb_kms, double mh) {
  if (!ctx || !m || !(teff > 0.0) || !(vturb_kms >= 0.0)) return fail(ctx, ATLASGPU_EINVAL, "model_set_params");
  cudaSetDevice(ctx->device);
  CK(cudaStreamSynchronize(ctx->stream));
  m->teff = teff;
  m->grav = pow(10.0, logg);
  m->vturb = vturb_kms;
  m->mh = mh;
  std::vector<double> v(m->kw, vturb_kms * 1.0e5);
  CK(cudaMemcpy(m->state + 6 * m->kw, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice));
  // the captured iteration holds the old scalars: capture again on next use
  if (m->gexec) cudaGraphExecDestroy(m->gexec);
  if (m->graph) cudaGraphDestroy(m->graph);
  m->gexec = nullptr;
  m->graph = nullptr;
  m->kapcont_done = false;
  return 0;
}

int atlasgpu_model_set_shard(atlasgpu_ctx* ctx, atlasgpu_model* m, int nu_first, int nu_last) {
  if (!ctx || !m || nu_first < 1 || nu_last < nu_first || nu_last > m->numnu)
    return fail(ctx, ATLASGPU_EINVAL, "model_set_shard: frequencies %d..%d outside 1..%d", nu_first, nu_last,
                m ? m->numnu : 0);
  cudaSetDevice(ctx->device);
  CK(cudaStreamSynchronize(ctx->stream));
  m->nu_first = nu_first;
  m->nu_last = nu_last;
  rt_shape(ctx, m);
  drop_graph(m);
  return 0;
}

int atlasgpu_model_set_sums_buffer(atlasgpu_ctx* ctx, atlasgpu_model* m, double* d_sums) {
  if (!ctx || !m) return fail(ctx, ATLASGPU_EINVAL, "model_set_sums_buffer: null");
  cudaSetDevice(ctx->device);
  CK(cudaStreamSynchronize(ctx->stream));
  m->ext_sums = d_sums;
  drop_graph(m);
  return 0;
}

int atlasgpu_model_iterate_begin(atlasgpu_ctx* ctx, atlasgpu_model* m) {
  if (!ctx || !m) return fail(ctx, ATLASGPU_EINVAL, "model_iterate_begin: null");
  cudaSetDevice(ctx->device);
  const int r = enqueue_begin(ctx, m, true);
  m->kapcont_done = true;
  return r;
}

int atlasgpu_model_iterate_end(atlasgpu_ctx* ctx, atlasgpu_model* m, double* maxerr) {
  if (!ctx || !m) return fail(ctx, ATLASGPU_EINVAL, "model_iterate_end: null");
  cudaSetDevice(ctx->device);
  int r;
  if ((r = enqueue_finish(ctx, m, true))) return r;
  double e = 0.0;
  CK(cudaMemcpyAsync(&e, m->maxerr_dev, sizeof e, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  if (maxerr) *maxerr = e;
  if (!(e == e)) return fail(ctx, ATLASGPU_ENONFINITE, "model_iterate_end: FLXERR is not finite");
  return 0;
}

int atlasgpu_model_destroy(atlasgpu_ctx* ctx, atlasgpu_model* m) {
  if (!m) return ATLASGPU_EINVAL;
  if (ctx) {
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
  }
  if (m->gexec) cudaGraphExecDestroy(m->gexec);
  if (m->graph) cudaGraphDestroy(m->graph);
  void* ps[] = {m->state, m->ms, m->xnfdop, m->dopple, m->xne_eos, m->txnxn, m->hkt, m->hckt, m->rho, m->cc,
                m->acont, m->sigmac,
                m->waveset, m->rcoset, m->cutwave, m->tabcont, m->iwavetab, m->linedata, m->lines, m->xl,
                m->xfix, m->fscale, m->funscale, m->cgfmax,
                m->partial, m->rt_rec, m->sum, m->hsurf, m->h0, m->h1, m->h2, m->hf, m->ross, m->R, m->iter_dev,
                m->maxerr_dev, m->cnt};
  for (void* p : ps)
    if (p) cudaFree(p);
  delete m;
  return ATLASGPU_OK;
}

double atlasgpu_fp64_peak_tflops(atlasgpu_ctx* ctx) {
  if (!ctx) return -1.0;
  cudaSetDevice(ctx->device);
  double* d;
  if (bufT(ctx, "peak_out", 1, &d)) return -1.0;
  const int iters = 4096, threads = 256, blocks = ctx->nsm * 8;
  k_fp64_fma<<<blocks, threads, 0, ctx->stream>>>(d, 64);  // warm-up
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, ctx->stream);
  k_fp64_fma<<<blocks, threads, 0, ctx->stream>>>(d, iters);
  cudaEventRecord(b, ctx->stream);
  cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (cudaGetLastError() != cudaSuccess || ms <= 0.f) return -1.0;
  const double flops = 2.0 * 8.0 * iters * (double)threads * blocks;
  return flops / (ms * 1e-3) / 1e12;
}

double atlasgpu_u64_atomic_peak(atlasgpu_ctx* ctx) {
  if (!ctx) return -1.0;
  cudaSetDevice(ctx->device);
  const size_t nwords = (size_t)1 << 23;  // 64 MB: LINOP1's fixed-point words of one model
  unsigned long long* w;
  if (bufT(ctx, "atom_peak", nwords, &w)) return -1.0;
  const int iters = 256, threads = 256, blocks = ctx->nsm * 8;
  k_u64_atomics<<<blocks, threads, 0, ctx->stream>>>(w, nwords, 16);  // warm-up
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, ctx->stream);
  k_u64_atomics<<<blocks, threads, 0, ctx->stream>>>(w, nwords, iters);
  cudaEventRecord(b, ctx->stream);
  cudaEventSynchronize(b);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (cudaGetLastError() != cudaSuccess || ms <= 0.f) return -1.0;
  return (double)iters * threads * blocks / (ms * 1e-3) / 1e9;
}

}  // extern "C"
