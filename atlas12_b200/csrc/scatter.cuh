// scatter.cuh -- JOSH's 51x51 scattering systems of many frequencies (FP64).
//
// The RT pass and the SYNTHE spectrum prepare one record per system (XALPHA,
// XSBAR and a solve flag, `stride` doubles apart) and solve them here, in two
// launches that split the systems by their contraction bound.  Both launches
// read the same flags and form the bound the same way.
//
// The system X = (1 - XALPHA) XSBAR + XALPHA (COEFJ X) is a
// contraction with factor q = max_l XALPHA(l) sum_m |COEFJ(l,m)| (the
// infinity norm of diag(XALPHA) COEFJ).  Where q <= kScatterSeriesQ
// its Neumann series is summed instead of eliminating: K steps of
// X <- (1 - XALPHA) XSBAR + XALPHA (COEFJ X) from X = (1 - XALPHA) XSBAR
// leave an error of at most q^(K+1) |X|, and K is taken so that
// q^(K+1) <= 2^-60, far below the rounding of the elimination itself (the
// two solutions agree to rounding).  A step is one matrix-vector product
// with no sequential dependence between rows and one barrier, against the
// elimination's 50 dependent pivot steps, so the series is cheaper up to
// q ~ 0.5.  Systems with larger q (strongly scattering layers) are
// eliminated as SOLVIT does.
#pragma once
#include "josh.cuh"

namespace atlasgpu {

// Records of n systems: system i at rec + i * stride, the 51-point vectors at
// the offsets xalpha, xsbar, xs, the flag (1: solve) at solve; per: systems
// of one group (consecutive).  work (timed launches only, else null):
// [0] systems eliminated, [1] systems summed as a series, [2] series steps.
struct ScatterArgs {
  const JoshOps* ops;
  double* rec;
  int stride, xalpha, xsbar, xs, solve, n, per;
  unsigned long long* work;
};

constexpr int kScatterGroups = 2;  // pair groups per CTA
constexpr int kScatterThreads = kScatterGroups * PairG::N;
constexpr int kScatterSolveMinBlocks = 4;  // 8 systems per SM (128 registers per thread)
constexpr double kScatterSeriesQ = 0.5;
constexpr int kScatterMaxSteps = 64;

struct ScatterWS {
  double xs[kNx], xsbar[kNx], xalpha[kNx], piv[kNx];
  double rowabs[kNx];  // row sums of |COEFJ| (the contraction bound's factors)
  double red[8];
  unsigned pk[4][3];
  alignas(16) double U[kNx * (kNx + 1)];
};
__host__ __device__ inline size_t scatter_smem_bytes() { return kScatterGroups * sizeof(ScatterWS); }

__device__ __forceinline__ int scatter_series_steps(double q) {
  if (!(q > 0.0)) return 1;
  const int k = (int)ceil(-60.0 * 0.6931471805599453 / log(q)) - 1;
  return k < 1 ? 1 : (k > kScatterMaxSteps ? kScatterMaxSteps : k);
}

// A system's result: XS, or with kSurf the surface flux HNU(1) = sum
// CH_J max(XS, 1e-37) (IFSURF = 1, atlas12_modules.f90:18571-18590) in XS's first word.
template <bool kSurf>
__device__ __forceinline__ void scatter_store(PairG& g, const ScatterArgs& a, double* rec, double x) {
  if (kSurf) {
    const double h = g.sum(g.r < kNx ? a.ops->ch[g.r] * fmax(x, 1.0e-37) : 0.0);
    if (g.r == 0) rec[a.xs] = h;
  } else if (g.r < kNx) {
    rec[a.xs + g.r] = x;
  }
}

template <bool kSurf>
static __device__ __forceinline__ void scatter_solve_body(const ScatterArgs& a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int gid = threadIdx.x / PairG::N;
  ScatterWS& S = reinterpret_cast<ScatterWS*>(smem_raw)[gid];
  PairG g(threadIdx.x % PairG::N, 1 + gid, S.red);
  const JoshOps& ops = *a.ops;
  const int i0 = (blockIdx.x * kScatterGroups + gid) * a.per, i1 = min(i0 + a.per, a.n);
  for (int l = g.r; l < kNx; l += PairG::N) {
    double r = 0.0;
    for (int m = 0; m < kNx; ++m) r += fabs(ops.coefj[m * kNx + l]);
    S.rowabs[l] = r;
  }
  g.sync();
  unsigned long long nelim = 0;
  for (int i = i0; i < i1; ++i) {
    double* rec = a.rec + (size_t)i * a.stride;
    if (rec[a.solve] != 1.0) continue;  // the same word for the whole group
    double qv = 0.0;
    for (int l = g.r; l < kNx; l += PairG::N) {
      const double xa = rec[a.xalpha + l];
      S.xalpha[l] = xa;
      S.xsbar[l] = rec[a.xsbar + l];
      qv = fmax(qv, xa * S.rowabs[l]);
    }
    const double q = g.max(qv);  // (its barrier also publishes XALPHA, XSBAR)
    if (q <= kScatterSeriesQ) continue;  // summed by scatter_series_body
    solve_scatter(g, ops, S, S.U);
    ++nelim;
    scatter_store<kSurf>(g, a, rec, g.r < kNx ? S.xs[g.r] : 0.0);
    g.sync();
  }
  if (a.work && g.r == 0 && nelim) atomicAdd(a.work, nelim);
}

// The Neumann series of the systems with q <= kScatterSeriesQ: thread l of a
// pair group keeps row l of COEFJ in registers for the whole launch (it is the
// same for every system), so a step is 51 FMAs on registers and the
// broadcast reads of X from shared memory, with no loads of COEFJ.  Sum k of
// the four partial sums takes the terms m = k, k+4, ... in that order; q is
// formed as in scatter_solve_body, so the two split the systems the same
// way.  (The series inside the elimination's kernel, reading COEFJ from L1 every step,
// took 2.6k cycles per step at eight groups per SM.)
constexpr int kScatterSeriesMinBlocks = 3;
struct ScatterSeriesWS {
  alignas(16) double xa[kNx + 1];
  alignas(16) double xb[kNx + 1];
  double red[8];
};

template <bool kSurf>
static __device__ __forceinline__ void scatter_series_body(const ScatterArgs& a) {
  __shared__ ScatterSeriesWS s_ws[kScatterGroups];
  const int gid = threadIdx.x / PairG::N;
  ScatterSeriesWS& S = s_ws[gid];
  PairG g(threadIdx.x % PairG::N, 1 + gid, S.red);
  const JoshOps& ops = *a.ops;
  const int l = g.r;
  const bool own = l < kNx;
  double c[kNx];
  double rowabs = 0.0;
#pragma unroll
  for (int m = 0; m < kNx; ++m) c[m] = own ? ops.coefj[m * kNx + l] : 0.0;
  for (int m = 0; m < kNx; ++m) rowabs += fabs(own ? ops.coefj[m * kNx + l] : 0.0);
  const int i0 = (blockIdx.x * kScatterGroups + gid) * a.per, i1 = min(i0 + a.per, a.n);
  unsigned long long nseries = 0, nsteps = 0;
  for (int i = i0; i < i1; ++i) {
    double* rec = a.rec + (size_t)i * a.stride;
    if (rec[a.solve] != 1.0) continue;  // the same word for the whole group
    const double al = own ? rec[a.xalpha + l] : 0.0;
    const double xb = own ? rec[a.xsbar + l] : 0.0;
    double qv = 0.0;
    if (own) qv = fmax(qv, al * rowabs);
    const double q = g.max(qv);
    if (q > kScatterSeriesQ) continue;  // eliminated by scatter_solve_body
    const int K = scatter_series_steps(q);
    const double b = own ? (1.0 - al) * xb : 0.0;
    double* cur = S.xa;
    double* nxt = S.xb;
    if (own) cur[l] = b;
    for (int k = 0; k < K; ++k) {
      g.sync();
      if (own) {
        double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int m = 0; m < kNx; ++m) s4[m & 3] = s4[m & 3] + c[m] * cur[m];
        nxt[l] = b + al * ((s4[0] + s4[1]) + (s4[2] + s4[3]));
      }
      double* t = cur;
      cur = nxt;
      nxt = t;
    }
    g.sync();
    scatter_store<kSurf>(g, a, rec, own ? cur[l] : 0.0);
    ++nseries;
    nsteps += K;
  }
  if (a.work && g.r == 0 && nseries) {
    atomicAdd(a.work + 1, nseries);
    atomicAdd(a.work + 2, nsteps);
  }
}

}  // namespace atlasgpu
