// scatter.cuh -- JOSH's 51x51 scattering systems of many frequencies (FP64).
//
// The RT pass and the SYNTHE spectrum prepare one record per system (XALPHA,
// XSBAR and a solve flag, `stride` doubles apart) and solve them here, in two
// launches: scatter_series_body sums the Neumann series of every system
// it settles, scatter_solve_body eliminates what is left as SOLVIT does.
//
// X = b + M X with b = (1 - XALPHA) XSBAR and M = diag(XALPHA) COEFJ is summed
// as X = sum d_k, d_0 = b, d_(k+1) = M d_k.  A system is settled
//   * by norm: q^(k+1) <= 2^-60 with q = max_l XALPHA(l) sum_m |COEFJ(l,m)| <= 1/2
//     (the rest is at most q^(k+1) |X|), or
//   * by its residual, which is the next increment: b + M X - X = d_(k+1), so the
//     error is (I - M)^-1 d_(k+1), at most |d_(k+1)| / (1 - q); settled when
//     d_(k+1) <= 2^-60 (1 - q) X in every row, q < 1.
// Both bounds are in the infinity norm, and far below the elimination's rounding.
// The norm bound counts the strongly scattering surface rows as if they fed
// themselves; they feed on deeper ones with small XALPHA, and the spectral
// radius of M is far smaller (0.04 where q = 0.49 in a solar spectrum at
// 400 nm).  Measured, the 83,800 systems of a 35 nm spectrum: 1.32 ms one system
// at a time from broadcast loads, 1.17 ms by matrix instructions with the norm
// bound alone, 0.38 ms with both.
// What 32 steps do not settle (spectral radius above ~0.27 at q > 1/2) is listed
// and eliminated.  The list spreads those systems, which are neighbours in
// frequency, over the GPU.  More steps hold the whole group of a slow system:
// 64 and 192 steps, or a second round of up to 192 for the left-overs in groups
// of their own, made the scattering stage of a 32-slot iteration 9.8, 15.7 and
// 10.7 ms against 8.8 with 32.
#pragma once
#include "josh.cuh"

namespace atlasgpu {

// Records of n systems: system i at rec + i * stride, the 51-point vectors at
// the offsets xalpha, xsbar, xs, the flag (1: solve) at solve; per_series:
// (consecutive) systems of one group of the series.  left, *nleft: the systems
// the series leaves over (zeroed by scatter_reset before it).  work (timed launches only, else
// null): [0] systems eliminated, [1] systems summed as a series, [2] series steps.
struct ScatterArgs {
  const JoshOps* ops;
  double* rec;
  int stride, xalpha, xsbar, xs, solve, n, per_series;
  int* left;
  unsigned* nleft;
  unsigned long long* work;
};
// doubles of a record buffer for cap systems, the list behind the records
__host__ __device__ inline size_t scatter_rec_doubles(size_t cap, size_t stride) { return cap * stride + (cap + 1) / 2 + 1; }
__host__ __device__ inline void scatter_lists(ScatterArgs& a, size_t cap) {
  a.nleft = reinterpret_cast<unsigned*>(a.rec + cap * a.stride);
  a.left = reinterpret_cast<int*>(a.nleft + 2);
}
// by one thread of the launch before the series
__device__ __forceinline__ void scatter_reset(const ScatterArgs& a) { *a.nleft = 0; }

constexpr int kScatterGroups = 2;  // pair groups per CTA
constexpr int kScatterThreads = kScatterGroups * PairG::N;
constexpr int kScatterSolveMinBlocks = 4;  // 8 systems per SM (128 registers per thread)
constexpr double kScatterSeriesQ = 0.5;  // largest q that is settled by norm
constexpr int kScatterMaxSteps = 64;     // ... within this many steps
constexpr int kScatterTrySteps = 32;      // most steps where only the residual can tell

struct ScatterWS {
  double xs[kNx], xsbar[kNx], xalpha[kNx], piv[kNx];
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
  const int n = (int)*a.nleft;
  unsigned long long nelim = 0;
  for (int i = blockIdx.x * kScatterGroups + gid; i < n; i += gridDim.x * kScatterGroups) {
    double* rec = a.rec + (size_t)a.left[i] * a.stride;
    for (int l = g.r; l < kNx; l += PairG::N) {
      S.xalpha[l] = rec[a.xalpha + l];
      S.xsbar[l] = rec[a.xsbar + l];
    }
    g.sync();
    solve_scatter(g, ops, S, S.U);
    ++nelim;
    scatter_store<kSurf>(g, a, rec, g.r < kNx ? S.xs[g.r] : 0.0);
    g.sync();
  }
  if (a.work && g.r == 0 && nelim) atomicAdd(a.work, nelim);
}

// The series, eight systems at a time by a pair of warps: a step is the product
// of COEFJ (51 x 51, padded to 56 x 52) with the eight vectors (52 x 8), in FP64
// matrix instructions (m8n8k4, which reach the FP64 pipe's 64 multiply-adds per
// clock and SM from one warp per scheduler).  COEFJ's fragments stay in
// registers for the whole launch, warp 0 of the pair holding rows 0..31 and
// warp 1 rows 32..55; the vectors go through shared memory once per step
// ([row][system]: fragment loads and result stores are both conflict-free).
// Bounded by the FP64 pipe: 23.3k multiply-adds per step of eight systems.
// A group runs the largest step count of its eight: further steps only add
// ever smaller terms.
constexpr int kScatterSeriesMinBlocks = 3;
constexpr int kSeriesN = 8;                       // systems per group
constexpr int kSeriesRows = 56, kSeriesK = 13;    // padded rows, 4-wide slices of the 52 columns
constexpr int kSeriesTiles = 4;                   // 8-row tiles of warp 0 (warp 1 has three)
struct ScatterSeriesWS {
  alignas(16) double x[2][kSeriesRows][kSeriesN];
  double part[3][2][kSeriesN];  // the two warps' parts of three reductions over rows (bound, settled, surface flux)
  int done[2][2];               // by parity of the step: a warp's rows are settled
};

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Launch shape of the series over n systems with 1/nb of the GPU: whole groups
// of eight, about two resident waves of warp pairs (six per SM at 168 registers).
inline int scatter_series_per(int n, int nsm, int nb) {
  const int units = nsm * 2 * kScatterSeriesMinBlocks * kScatterGroups / (nb > 0 ? nb : 1);
  const int batches = (n + kSeriesN - 1) / kSeriesN;
  return kSeriesN * ((batches + (units > 0 ? units : 1) - 1) / (units > 0 ? units : 1));
}
inline int scatter_series_blocks(int n, int per) {
  return ((n + per - 1) / per + kScatterGroups - 1) / kScatterGroups;
}

// CTAs of the elimination (they walk the list with a grid stride; one without work ends at once)
inline int scatter_solve_blocks(int n, int nsm) {
  const int need = (n + kScatterGroups - 1) / kScatterGroups, most = nsm * kScatterSolveMinBlocks;
  return need < most ? need : most;
}

template <bool kSurf>
static __device__ __forceinline__ void scatter_series_body(const ScatterArgs& a) {
  __shared__ ScatterSeriesWS s_ws[kScatterGroups];
  const JoshOps& ops = *a.ops;
  const int gid = threadIdx.x / PairG::N;
  ScatterSeriesWS& S = s_ws[gid];
  PairG g(threadIdx.x % PairG::N, 1 + gid, nullptr);
  const int lane = g.r & 31, warp = g.r >> 5;
  const int tr = lane >> 2, tc = lane & 3;  // result fragment: row tr of a tile, systems 2 tc and 2 tc + 1
  const int ntile = warp == 0 ? kSeriesTiles : kSeriesRows / 8 - kSeriesTiles;
  const int row0 = warp * kSeriesTiles * 8 + tr;  // this lane's row of tile t: row0 + 8 t
  double cf[kSeriesTiles][kSeriesK];
#pragma unroll
  for (int t = 0; t < kSeriesTiles; ++t) {
    const int row = row0 + 8 * t;
#pragma unroll
    for (int k = 0; k < kSeriesK; ++k) {
      const int m = 4 * k + tc;
      cf[t][k] = (t < ntile && row < kNx && m < kNx) ? ops.coefj[m * kNx + row] : 0.0;
    }
  }
  const int i0 = (blockIdx.x * kScatterGroups + gid) * a.per_series, i1 = min(i0 + a.per_series, a.n);
  unsigned long long nseries = 0, nsteps = 0;
  for (int ib = i0; ib < i1; ib += kSeriesN) {
    // the lane's two systems: XALPHA and d_0 of its rows, 0 where there is nothing to sum
    bool want[2];
    double al[kSeriesTiles][2], x[kSeriesTiles][2], qv[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = ib + 2 * tc + e;
      const double* rec = a.rec + (size_t)i * a.stride;
      want[e] = i < i1 && rec[a.solve] == 1.0;
#pragma unroll
      for (int t = 0; t < kSeriesTiles; ++t) {
        const int row = row0 + 8 * t;
        const bool on = want[e] && t < ntile && row < kNx;
        al[t][e] = on ? rec[a.xalpha + row] : 0.0;
        x[t][e] = on ? (1.0 - al[t][e]) * rec[a.xsbar + row] : 0.0;
        if (on) qv[e] = fmax(qv[e], al[t][e] * ops.rowabs[row]);
      }
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) qv[e] = fmax(qv[e], __shfl_xor_sync(0xffffffffu, qv[e], o));
      if (tr == 0) S.part[0][warp][2 * tc + e] = qv[e];
    }
    g.sync();
    int cap[2], K = 0;  // steps after which the system is settled by norm; else given up
    bool norm[2], had[2] = {want[0], want[1]};
    double tol[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double q = fmax(S.part[0][0][2 * tc + e], S.part[0][1][2 * tc + e]);
      norm[e] = !(q > kScatterSeriesQ);
      want[e] = want[e] && !(q >= 1.0);
      tol[e] = 0x1p-60 * (1.0 - q);
      cap[e] = !want[e] ? 0 : (norm[e] ? scatter_series_steps(q) : kScatterTrySteps);
      K = max(K, cap[e]);
#pragma unroll
      for (int t = 0; t < kSeriesTiles; ++t)
        if (!want[e]) al[t][e] = x[t][e] = 0.0;
    }
    K = __reduce_max_sync(0xffffffffu, K);  // the same for both warps
#pragma unroll
    for (int t = 0; t < kSeriesTiles; ++t)
      if (t < ntile) *reinterpret_cast<double2*>(&S.x[0][row0 + 8 * t][2 * tc]) = make_double2(x[t][0], x[t][1]);
    bool ok[2] = {true, true};  // this lane's rows are settled by the residual
    int k = 0;
    for (; k < K; ++k) {
      g.sync();
      if (k > 0 && S.done[k & 1][0] && S.done[k & 1][1]) break;
      const double(*cur)[kSeriesN] = S.x[k & 1];
      double y[kSeriesTiles][2];
#pragma unroll
      for (int t = 0; t < kSeriesTiles; ++t) y[t][0] = y[t][1] = 0.0;
#pragma unroll
      for (int kk = 0; kk < kSeriesK; ++kk) {
        const double bf = cur[4 * kk + tc][tr];
#pragma unroll
        for (int t = 0; t < kSeriesTiles; ++t)
          if (t < ntile) dmma(y[t][0], y[t][1], cf[t][kk], bf);
      }
      ok[0] = ok[1] = true;
#pragma unroll
      for (int t = 0; t < kSeriesTiles; ++t) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double dn = al[t][e] * y[t][e];
          x[t][e] += dn;
          ok[e] = ok[e] && fabs(dn) <= tol[e] * fabs(x[t][e]);
          y[t][e] = dn;
        }
        if (t < ntile)
          *reinterpret_cast<double2*>(&S.x[(k + 1) & 1][row0 + 8 * t][2 * tc]) = make_double2(y[t][0], y[t][1]);
      }
      const int done = __all_sync(0xffffffffu, (ok[0] || k + 1 >= cap[0]) && (ok[1] || k + 1 >= cap[1]));
      if (lane == 0) S.done[(k + 1) & 1][warp] = done;
    }
    // settled: by norm within the steps run, or by the residual in every row
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const unsigned rows = 0x11111111u << tc;  // the lanes with this lane's systems
      const bool all = (__ballot_sync(0xffffffffu, ok[e]) & rows) == rows;
      if (tr == 0) S.part[1][warp][2 * tc + e] = all ? 1.0 : 0.0;
    }
    g.sync();
#pragma unroll
    for (int e = 0; e < 2; ++e)
      want[e] = want[e] && ((norm[e] && k >= cap[e]) ||
                            (S.part[1][0][2 * tc + e] != 0.0 && S.part[1][1][2 * tc + e] != 0.0));
    if (a.work && warp == 0 && tr == 0) {
      nseries += (unsigned)want[0] + (unsigned)want[1];
      nsteps += (unsigned long long)k * ((unsigned)want[0] + (unsigned)want[1]);
    }
    if (warp == 0 && tr == 0) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (had[e] && !want[e]) a.left[atomicAdd(a.nleft, 1u)] = ib + 2 * tc + e;
    }
    if (kSurf) {
      double h[2] = {0.0, 0.0};
#pragma unroll
      for (int t = 0; t < kSeriesTiles; ++t) {
        const int row = row0 + 8 * t;
        if (t >= ntile || row >= kNx) continue;
        const double ch = ops.ch[row];
        h[0] += ch * fmax(x[t][0], 1.0e-37);
        h[1] += ch * fmax(x[t][1], 1.0e-37);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) h[e] += __shfl_xor_sync(0xffffffffu, h[e], o);
        if (tr == 0) S.part[2][warp][2 * tc + e] = h[e];
      }
      g.sync();
      if (warp == 0 && tr == 0) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (want[e])
            a.rec[(size_t)(ib + 2 * tc + e) * a.stride + a.xs] = S.part[2][0][2 * tc + e] + S.part[2][1][2 * tc + e];
      }
      g.sync();
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (want[e]) {
          double* rec = a.rec + (size_t)(ib + 2 * tc + e) * a.stride + a.xs;
#pragma unroll
          for (int t = 0; t < kSeriesTiles; ++t)
            if (t < ntile && row0 + 8 * t < kNx) rec[row0 + 8 * t] = x[t][e];
        }
      g.sync();
    }
  }
  if (a.work && nseries) {
    atomicAdd(a.work + 1, nseries);
    atomicAdd(a.work + 2, nsteps);
  }
}

}  // namespace atlasgpu
