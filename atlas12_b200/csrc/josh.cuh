// josh.cuh -- cooperative JOSH radiative transfer (FP64) for sm_100a.
//
// A thread group solves one frequency: either one warp (WarpG) or a pair of
// warps (PairG, 64 threads synchronised by a named barrier).  Depth vectors
// (<= kKwMax) live in the group's shared-memory workspace; threads split
// depths, grid points, matrix rows or columns.  Every routine restates the
// reference formula for each output element (atlas12_modules.f90):
//   PARCOE :5358-5434, INTEG :5293-5324, DERIV :5228-5266, MAP1 :5570-5692,
//   SOLVIT :5739-5847, JOSH :18398-18776.
// Every output point of INTEG, DERIV and MAP1 is computed on its own, from the
// interval it lies in (the Newton form below).
//
// The 51x51 scattering system: a pair group keeps one matrix row per thread
// in registers and writes only the pivot rows to shared memory, which takes
// the row updates off the shared-memory pipe.
#pragma once
#include "common.cuh"

namespace atlasgpu {

// ---------------------------------------------------------------- groups
struct WarpG {
  static constexpr int N = 32;
  int r;  // lane
  __device__ explicit WarpG(int lane) : r(lane) {}
  __device__ __forceinline__ void sync() const { __syncwarp(0xffffffffu); }
  __device__ __forceinline__ double max(double v) { return warp_max(v); }
  __device__ __forceinline__ double sum(double v) { return warp_sum(v); }
  __device__ __forceinline__ bool any(bool p) { return __any_sync(0xffffffffu, p); }
};

// NW warps on named barrier `bar`; red = 2*NW doubles of the group's shared
// scratch (one slot per warp and parity, alternated so one barrier per
// reduction suffices: a slot is rewritten only after every thread has passed
// the barrier of the reduction in between).  Warp partials are combined in
// warp order, so the result does not depend on scheduling.
template <int NW>
struct MultiG {
  static constexpr int N = 32 * NW;
  int r;  // 0..N-1
  int bar;
  double* red;
  int par;
  __device__ MultiG(int rank, int barrier, double* scratch) : r(rank), bar(barrier), red(scratch), par(0) {}
  __device__ __forceinline__ void sync() const {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(N) : "memory");
  }
  __device__ __forceinline__ double sum(double v) {
    v = warp_sum(v);
    if ((r & 31) == 0) red[par * NW + (r >> 5)] = v;
    sync();
    double s = red[par * NW];
#pragma unroll
    for (int w = 1; w < NW; ++w) s += red[par * NW + w];
    par ^= 1;
    return s;
  }
  __device__ __forceinline__ double max(double v) {
    v = warp_max(v);
    if ((r & 31) == 0) red[par * NW + (r >> 5)] = v;
    sync();
    double s = red[par * NW];
#pragma unroll
    for (int w = 1; w < NW; ++w) s = fmax(s, red[par * NW + w]);
    par ^= 1;
    return s;
  }
  __device__ __forceinline__ bool any(bool p) { return max(__any_sync(0xffffffffu, p) ? 1.0 : 0.0) > 0.0; }
};
using PairG = MultiG<2>;

struct JoshWS {
  double xs[kNx], xsbar[kNx], xalpha[kNx], xw[kNx];
  double abtot[kKwMax], alpha[kKwMax], snubar[kKwMax], taunu[kKwMax];
  double rd[kKwMax], r2[kKwMax];  // reciprocal differences of TAUNU (recip_range)
  double t1[kKwMax];              // scratch (INTEG's terms)
  double red[8];                  // group reductions (multi-warp groups)
  double piv[kNx];                // pivots of the elimination without interchanges
  int last;                       // MAP1 bracket of the last grid point
  unsigned pk[4][3];              // pivot key exchange between a group's warps
};

// Full-solution extras for IFSURF = 0 (ATLAS)
struct JoshWSFull {
  double snu[kKwMax], hnu[kKwMax], jmins[kKwMax], jnu[kKwMax], bnu[kKwMax];
  double knu1;
  int maxj;
};

// ---------------------------------------------------------------- interpolation
// PARCOE, INTEG, DERIV and MAP1 in Newton form.  On the interval
// [x(i), x(i+1)] both of the reference's parabolas (through i-1, i, i+1 and
// through i, i+1, i+2) pass through its two end points, so any blend of them is
//   f(i) + (v - x(i)) (slope(i) + (v - x(i+1)) q),
// q the same blend of their second divided differences.  MAP1's reuse of the
// previous forward parabola as the next backward one gives the same parabola,
// so no state is carried from output to output.  A value costs one division
// (the blend) where the reference's A, B, C form costs eleven, and with the
// reciprocal differences of the grid given (recip_range, shared by every
// function on the grid) none for the differences.  The A + (B + C v) v form loses
// digits to cancellation where v is far from 0; this one does not.
// (FP64 divisions bound the RT pass's prepare and finish stages: with the
// reference's form they took 0.18 and 0.78 ms per 30,000 x 72 model-iteration.)

// Reciprocal differences of a grid: rd(i) = 1/(x(i+1) - x(i)), i < n-1, and
// r2(i) = 1/(x(i+1) - x(i-1)), 0 < i < n-1.  The caller synchronises.
__device__ __forceinline__ void recip_range(int r, int step, const double* x, double* rd, double* r2, int n) {
  for (int i = r; i < n - 1; i += step) {
    rd[i] = 1.0 / (x[i + 1] - x[i]);
    if (i > 0) r2[i] = 1.0 / (x[i + 1] - x[i - 1]);
  }
}

// Reciprocals on the fly, for a grid that only one function is mapped on
struct GridX {
  const double* x;
  __device__ __forceinline__ double rd(int i) const { return 1.0 / (x[i + 1] - x[i]); }
  __device__ __forceinline__ double r2(int i) const { return 1.0 / (x[i + 1] - x[i - 1]); }
};
// ... or from recip_range's arrays
struct GridP {
  const double *rdp, *r2p;
  __device__ __forceinline__ double rd(int i) const { return rdp[i]; }
  __device__ __forceinline__ double r2(int i) const { return r2p[i]; }
};

// PARCOE's and MAP1's blend of the backward and forward second differences
__device__ __forceinline__ double blend_curv(double cb, double cf) {
  double wt = 0.0;
  if (fabs(cf) != 0.0) wt = fabs(cf) / (fabs(cf) + fabs(cb));
  return cf + wt * (cb - cf);
}

// fint = running parabolic integral of f over x, fint[0] = start (INTEG over
// PARCOE's coefficients: linear on intervals 0..2 and the last, blended
// parabolas between).  term: n doubles of scratch.  The running sum is formed
// by the group's first warp, each lane a run of consecutive intervals, and a
// scan of the lanes' sums (the one-thread sum was 71 dependent additions).
template <class G, class R>
__device__ inline void g_integ(G& g, const double* x, const double* f, double* fint, int n, double start,
                               double* term, R gr) {
  for (int i = g.r; i < n - 1; i += G::N) {
    const double h = x[i + 1] - x[i];
    double t = 0.5 * h * (f[i] + f[i + 1]);
    if (i >= 3 && i <= n - 3) {
      const double s = (f[i + 1] - f[i]) * gr.rd(i);
      const double cb = (s - (f[i] - f[i - 1]) * gr.rd(i - 1)) * gr.r2(i);
      const double cf = ((f[i + 2] - f[i + 1]) * gr.rd(i + 1) - s) * gr.r2(i + 1);
      t -= blend_curv(cb, cf) * (h * h * h) * (1.0 / 6.0);
    }
    term[i] = t;
  }
  g.sync();
  if (g.r < 32) {
    const int per = (n - 1 + 31) >> 5, i0 = g.r * per, i1 = min(i0 + per, n - 1);
    double own = 0.0;
    for (int i = i0; i < i1; ++i) own += term[i];
    double run = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, run, o);
      if (g.r >= o) run += v;
    }
    run = __shfl_up_sync(0xffffffffu, run, 1);
    run = g.r == 0 ? start : start + run;
    if (g.r == 0) fint[0] = start;
    for (int i = i0; i < i1; ++i) {
      run += term[i];
      fint[i + 1] = run;
    }
  }
  g.sync();
}
template <class G, class WS>
__device__ inline void g_integ(G& g, const double* x, const double* f, double* fint, int n, double start, WS& ws) {
  g_integ(g, x, f, fint, n, start, ws.t1, GridX{x});
}

// ---------------------------------------------------------------- DERIV
// DERIV at point j of the n points (x, f): the end points' slopes, and the
// tangent of the mean of the two slopes' angles (in the reference's scaled
// variables) between them.  tan of the mean from one quotient instead of the
// reference's three.
template <class R>
__device__ __forceinline__ double deriv_at(const double* x, const double* f, int n, int j, R gr) {
  if (j == 0) return (f[1] - f[0]) * gr.rd(0);
  if (j == n - 1) return (f[n - 1] - f[n - 2]) * gr.rd(n - 2);
  const double s = copysign(1.0, x[1] - x[0]);
  const double top = fmax(fmax(fabs(f[j - 1]), fabs(f[j])), fabs(f[j + 1])), ax = fabs(x[j]);
  const double rs = top == 0.0 ? 1.0 : ax / top;  // 1/SCALE, SCALE = top/|x| (1 where f is 0 around j)
  const double dr = (f[j + 1] - f[j]) * gr.rd(j) * rs;
  const double dl = (f[j] - f[j - 1]) * gr.rd(j - 1) * rs;
  const double er = s * sqrt(1.0 + dr * dr) + 1.0, el = s * sqrt(1.0 + dl * dl) + 1.0;
  return (dr * el + dl * er) / ((er * el - dr * dl) * rs);
}

// dfdx may alias f in callers
template <class G, class R>
__device__ __noinline__ void g_deriv_on(G g, const double* x, const double* f, double* dfdx, int n, R gr) {
  constexpr int C = (kKwMax + G::N - 1) / G::N;
  double v[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = g.r + c * G::N;
    if (j < n) v[c] = deriv_at(x, f, n, j, gr);
  }
  g.sync();
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = g.r + c * G::N;
    if (j < n) dfdx[j] = v[c];
  }
  g.sync();
}
template <class G>
__device__ __forceinline__ void g_deriv(G& g, const double* x, const double* f, double* dfdx, int n) {
  g_deriv_on(g, x, f, dfdx, n, GridX{x});
}

// ---------------------------------------------------------------- MAP1
// MAP1's bracket of v: L = min{L >= 2 : XOLD(L) > v} (1-based), nold+1 past the end
__device__ __forceinline__ int map1_bracket(const double* xo, int nold, double v) {
  int lo = 2, hi = nold + 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (xo[mid - 1] > v) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

// One output point of MAP1 with the differences its value needs, so that
// several functions on the same old grid share them: linear in the first two
// intervals and past the end, the backward parabola alone in the last
// interval, the blend elsewhere.
struct Map1At {
  int i, mode;  // interval (0-based lower point); 0 linear, 1 backward, 2 blended
  double v0, v1, rd0, rdm, rdp, r20, r2p;
  template <class R>
  __device__ __forceinline__ Map1At(const double* xo, int nold, int L, double v, R gr) {
    i = (L > nold ? nold : L) - 2;
    mode = (L <= 3 || L > nold) ? 0 : (L == nold ? 1 : 2);
    v0 = v - xo[i];
    v1 = v - xo[i + 1];
    rd0 = gr.rd(i);
    rdm = rdp = r20 = r2p = 0.0;
    if (mode >= 1) {
      rdm = gr.rd(i - 1);
      r20 = gr.r2(i);
    }
    if (mode == 2) {
      rdp = gr.rd(i + 1);
      r2p = gr.r2(i + 1);
    }
  }
  __device__ __forceinline__ double operator()(const double* fo) const {
    const double f0 = fo[i], f1 = fo[i + 1];
    const double s = (f1 - f0) * rd0;
    if (mode == 0) return f1 + v1 * s;
    double q = (s - (f0 - fo[i - 1]) * rdm) * r20;
    if (mode == 2) q = blend_curv(q, ((fo[i + 2] - f1) * rdp - s) * r2p);
    return f0 + v0 * (s + v1 * q);
  }
};

// Returns MAP1 (index of the last old interval used).  xnew ascending.
template <class G>
__device__ __noinline__ int g_map1_on(G g, const double* xo, const double* fo, int nold, const double* xn,
                                      double* fn, int nnew) {
  for (int k = g.r; k < nnew; k += G::N) {
    const double v = xn[k];
    fn[k] = Map1At(xo, nold, map1_bracket(xo, nold, v), v, GridX{xo})(fo);
  }
  const int L = map1_bracket(xo, nold, xn[nnew - 1]);
  g.sync();
  return (L > nold ? nold : L) - 1;
}
template <class G>
__device__ __forceinline__ int g_map1(G& g, const double* xo, const double* fo, int nold, const double* xn,
                                      double* fn, int nnew) {
  return g_map1_on(g, xo, fo, nold, xn, fn, nnew);
}

// ---------------------------------------------------------------- SOLVIT
constexpr double kPivotTol = 1.0e-30;

// Pivot-row traffic in 16-byte words: the row owner stores [1/pivot, a[1..]]
// and every pending row reads it back as double2 words (U rows are 16-byte
// aligned: 52 doubles per row on a 16-byte aligned base).  From step 26 on,
// only the first 26 entries of a shifted row can be nonzero (columns i..50
// and the rhs), so those steps move and update NW = 13 words instead of 26.
template <int NW = (kNx + 1) / 2>
__device__ __forceinline__ void store_pivot_row(double* ur, double rpiv, const double (&a)[kNx + 1]) {
  double2* u2 = reinterpret_cast<double2*>(ur);
  u2[0] = make_double2(rpiv, a[1]);
#pragma unroll
  for (int q = 1; q < NW; ++q) u2[q] = make_double2(a[2 * q], a[2 * q + 1]);
}

// a[t-1] = a[t] - l * ur[t] (t = 1..2NW-1), l = a[0] * ur[0]; the entry
// shifted in from beyond the stored words is zero (a[2NW-1] = 0)
template <int NW = (kNx + 1) / 2>
__device__ __forceinline__ void eliminate_shift(double (&a)[kNx + 1], const double* ur) {
  const double2* u2 = reinterpret_cast<const double2*>(ur);
  const double2 u0 = u2[0];
  const double l = a[0] * u0.x;
  a[0] = a[1] - l * u0.y;
#pragma unroll
  for (int q = 1; q < NW; ++q) {
    const double2 u = u2[q];
    a[2 * q - 1] = a[2 * q] - l * u.x;
    a[2 * q] = a[2 * q + 1] - l * u.y;
  }
  a[2 * NW - 1] = 0.0;
}

constexpr int kHalfStep = (kNx + 1) / 2;  // first step whose pending rows fit in half a row

// Back substitution from the stored pivot rows U (row k: U[k][0] = 1/pivot,
// U[k][t] = column k+t, the rhs at t = 51-k) by the group's first warp: lane
// q holds positions q and q+32, X(j) = B(j) * (1/pivot) is passed by shuffle
// and B(k) -= A(k,j) X(j) for k < j, in SOLVIT's order.  XS receives X.
__device__ __forceinline__ void u_back_substitute(int r, const double* U, double* xs) {
  constexpr int n = kNx, W = kNx + 1;
  if (r >= 32) return;
  const int k0 = r, k1 = r + 32;
  double b0 = U[k0 * W + (W - 1 - k0)];
  double b1 = k1 < n ? U[k1 * W + (W - 1 - k1)] : 0.0;
  for (int j = n - 1; j >= 0; --j) {
    const int src = j & 31;
    double x = (j < 32 ? b0 : b1) * U[j * W];
    x = __shfl_sync(0xffffffffu, x, src);
    if (r == src) xs[j] = x;
    if (k0 < j) b0 = b0 - U[k0 * W + (j - k0)] * x;
    if (k1 < j) b1 = b1 - U[k1 * W + (j - k1)] * x;
  }
}

// The same system by a pair group, thread r < 51 holding row r of
// [AMAT | rhs] in registers.  The elimination follows SOLVIT's arithmetic:
// the pivot of step i is the first maximum |A(k,i)| over the rows at
// positions i..50 (rows are swapped logically: each thread tracks the
// position of its row), the pivot is replaced by its reciprocal (clamped at
// 1e-30), multipliers are A(k,i) * (1/pivot), the right-hand side is
// eliminated with the same multipliers in step order, and back substitution
// runs column by column from the last.
// Each step shifts the pending rows one column left, so column i is always
// register a[0] and the loop over steps stays rolled (one short loop body
// instead of 51 unrolled steps).  The pivot row of step i is stored in
// U[i][0..51] (U[i][0] = 1/pivot, U[i][t] = column i+t, the rhs at t = 51-i)
// for the other rows' update and for the back substitution.
// The pivot search reduces a 64-bit key (|a| bits, then position) with
// redux.sync per warp and one exchange between the two warps.
template <class WS>
static __device__ __forceinline__ void scatter_solve(PairG& g, const JoshOps& ops, WS& ws, double* U) {
  constexpr int n = kNx, W = kNx + 1;
  constexpr unsigned FULL = 0xffffffffu;
  const bool own = g.r < n;
  double a[W];
  {
    const int l = own ? g.r : 0;
    const double xa = ws.xalpha[l];
#pragma unroll
    for (int m = 0; m < n; ++m) {
      double v = -xa * ops.coefj[m * kNx + l];
      if (l == m) v = v + 1.0;
      a[m] = v;
    }
    a[n] = (1.0 - xa) * ws.xsbar[l];
  }
  int pos = own ? g.r : n + 1;  // current row position
  bool done = !own;
  for (int i = 0; i < n - 1; ++i) {
    // (a) pivot: max |A(pos, i)| over pending rows, ties to the lowest position
    unsigned hi = 0u, lo = 0u;
    if (!done) {
      const unsigned long long bits = (unsigned long long)__double_as_longlong(fabs(a[0]));
      hi = (unsigned)(bits >> 32) + 1u;  // 0 marks rows already eliminated
      lo = (unsigned)bits;
    }
    const unsigned mhi = __reduce_max_sync(FULL, hi);
    const unsigned mlo = __reduce_max_sync(FULL, hi == mhi ? lo : 0u);
    const unsigned mpos =
        __reduce_min_sync(FULL, (hi != 0u && hi == mhi && lo == mlo) ? (unsigned)pos : 0xffffffffu);
    if ((g.r & 31) == 0) {
      ws.pk[g.r >> 5][0] = mhi;
      ws.pk[g.r >> 5][1] = mlo;
      ws.pk[g.r >> 5][2] = mpos;
    }
    g.sync();
    unsigned bpos;
    {
      const unsigned h0 = ws.pk[0][0], l0 = ws.pk[0][1], p0 = ws.pk[0][2];
      const unsigned h1 = ws.pk[1][0], l1 = ws.pk[1][1], p1 = ws.pk[1][2];
      const bool second = h1 > h0 || (h1 == h0 && (l1 > l0 || (l1 == l0 && p1 < p0)));
      bpos = second ? p1 : p0;
    }
    const bool me = !done && (unsigned)pos == bpos;
    // (b) the row at position i moves to the pivot's position
    if (!done && !me && pos == i) pos = (int)bpos;
    // (c) the pivot row, with its reciprocal pivot, to every thread
    double* ur = U + i * W;
    if (me) {
      double pv = a[0];
      if (fabs(pv) < kPivotTol) pv = copysign(kPivotTol, pv);
      if (i < kHalfStep) store_pivot_row(ur, 1.0 / pv, a);
      else store_pivot_row<kHalfStep / 2>(ur, 1.0 / pv, a);
      pos = i;
      done = true;
    }
    g.sync();
    // (d, e) multiplier and trailing update of the pending rows, shifted left
    if (!done) {
      if (i < kHalfStep) eliminate_shift(a, ur);
      else eliminate_shift<kHalfStep / 2>(a, ur);
    }
  }
  // the last pending row takes position n-1: column n-1 in a[0], rhs in a[1]
  if (!done) {
    pos = n - 1;
    double v = a[0];
    if (fabs(v) < kPivotTol) v = copysign(kPivotTol, v);
    U[(n - 1) * W] = 1.0 / v;
    U[(n - 1) * W + 1] = a[1];
  }
  g.sync();
  u_back_substitute(g.r, U, ws.xs);
  g.sync();
}

// Elimination without interchanges, checked: thread r < 51 holds row r,
// which becomes the pivot row at step r.  At step i every pending row
// compares its |A(k,i)| with the pivot |A(i,i)|; SOLVIT's first-maximum rule
// would pick another row only if some |A(k,i)| is strictly larger.  Returns
// false (the caller then redoes the system with interchanges) if that ever
// happened; otherwise the operations were exactly SOLVIT's, in its order.
// (For these systems it does not happen: AMAT is column diagonally dominant
// because the columns of COEFJ sum to at most 1 and XALPHA < 1.)
template <class WS>
static __device__ __forceinline__ bool scatter_solve_nopivot(PairG& g, const JoshOps& ops, WS& ws, double* U) {
  constexpr int n = kNx, W = kNx + 1;
  const bool own = g.r < n;
  double a[W];
  {
    const int l = own ? g.r : 0;
    const double xa = ws.xalpha[l];
#pragma unroll
    for (int m = 0; m < n; ++m) {
      double v = -xa * ops.coefj[m * kNx + l];
      if (l == m) v = v + 1.0;
      a[m] = v;
    }
    a[n] = (1.0 - xa) * ws.xsbar[l];
  }
  bool swap = false;
  for (int i = 0; i < n - 1; ++i) {
    double* ur = U + i * W;
    if (g.r == i) {
      ws.piv[i] = a[0];
      double pv = a[0];
      if (fabs(pv) < kPivotTol) pv = copysign(kPivotTol, pv);
      if (i < kHalfStep) store_pivot_row(ur, 1.0 / pv, a);
      else store_pivot_row<kHalfStep / 2>(ur, 1.0 / pv, a);
    }
    g.sync();
    if (own && g.r > i) {
      swap |= fabs(a[0]) > fabs(ws.piv[i]);
      if (i < kHalfStep) eliminate_shift(a, ur);
      else eliminate_shift<kHalfStep / 2>(a, ur);
    }
  }
  if (g.r == n - 1) {
    double v = a[0];
    if (fabs(v) < kPivotTol) v = copysign(kPivotTol, v);
    U[(n - 1) * W] = 1.0 / v;
    U[(n - 1) * W + 1] = a[1];
  }
  if (g.any(swap)) return false;
  u_back_substitute(g.r, U, ws.xs);
  g.sync();
  return true;
}


template <class WS>
__device__ __forceinline__ void solve_scatter(PairG& g, const JoshOps& ops, WS& ws, double* U) {
  if (!scatter_solve_nopivot(g, ops, ws, U)) scatter_solve(g, ops, ws, U);
}
// ---------------------------------------------------------------- JOSH
// JOSH in three parts, so that a caller may run them in separate launches
// (the ATLAS12 RT pass runs the 51x51 solve in its own kernel):
//   g_josh_prepare  TAUNU = INTEG(ABTOT dRHOX), MAXJ, and for MAXJ != 1 XSBAR
//                   and XALPHA on the 51-point grid with their floors
//                   (atlas12_modules.f90:18491-18570); solve = max XALPHA > 0,
//                   otherwise XS = XSBAR
//   solve_scatter   (I - diag(XALPHA) COEFJ) XS = (1 - XALPHA) XSBAR
//   g_josh_finish   XS floor, SNU = MAP1(XS), J/H/K from the operators mapped
//                   back onto the depths, the Eddington sweeps below MAXJ
//                   (:18571-18776)
// ws.abtot, ws.alpha and ws.snubar are formed by the caller (g_josh_fill).
template <class G, class WS>
__device__ inline void g_josh_fill(G& g, int nr, const double* acont, const double* aline, const double* sigmac,
                                   const double* sigmal, const double* scont, const double* sline, WS& ws) {
  for (int j = g.r; j < nr; j += G::N) {
    const double ab = acont[j] + aline[j] + sigmac[j] + sigmal[j];
    ws.abtot[j] = ab;
    ws.alpha[j] = (sigmac[j] + sigmal[j]) / ab;
    ws.snubar[j] = (acont[j] * scont[j] + aline[j] * sline[j]) / (acont[j] + aline[j]);
  }
  g.sync();
}

// The grids every frequency of a launch shares, with their reciprocal
// differences: RHOX and JOSH's 51-point tau grid.  One per CTA, in shared
// memory; josh_grid_load by all its threads (it synchronises the CTA).
struct JoshGrid {
  double rhox[kKwMax], rrd[kKwMax], rr2[kKwMax];
  double xtau[kNx], xrd[kNx], xr2[kNx];
  __device__ __forceinline__ GridP rho() const { return GridP{rrd, rr2}; }
  __device__ __forceinline__ GridP tau() const { return GridP{xrd, xr2}; }
};
__device__ __forceinline__ void josh_grid_load(JoshGrid& J, const JoshOps& ops, const double* rhox, int nr) {
  for (int j = threadIdx.x; j < nr; j += blockDim.x) J.rhox[j] = rhox[j];
  for (int l = threadIdx.x; l < kNx; l += blockDim.x) J.xtau[l] = ops.xtau[l];
  recip_range(threadIdx.x, blockDim.x, rhox, J.rrd, J.rr2, nr);
  recip_range(threadIdx.x, blockDim.x, ops.xtau, J.xrd, J.xr2, kNx);
  __syncthreads();
}

// mapped: the surface is optically thin enough for the 51-point grid (MAP1
// may still return MAXJ = 1 there, and IFSURF = 1 then takes H(1) from XS).
// Leaves TAUNU's reciprocal differences in ws.rd and ws.r2.
template <class G, class WS>
__device__ inline int g_josh_prepare(G& g, const JoshGrid& J, int nr, WS& ws, bool& mapped, bool& solve) {
  g_integ(g, J.rhox, ws.abtot, ws.taunu, nr, ws.abtot[0] * J.rhox[0], ws.rd, J.rho());
  recip_range(g.r, G::N, ws.taunu, ws.rd, ws.r2, nr);
  g.sync();
  solve = false;
  const double tau1 = ws.taunu[0];
  mapped = !(tau1 > J.xtau[kNx - 1]);
  if (!mapped) return 1;
  // SNUBAR and ALPHA onto the 51-point grid, one bracket and one set of
  // differences for both; the surface values above the first depth's TAU
  const GridP gr{ws.rd, ws.r2};
  double amax = -1.0;
  int last = 0;
  for (int l = g.r; l < kNx; l += G::N) {
    const double x = J.xtau[l];
    last = map1_bracket(ws.taunu, nr, x);
    double xa, xb;
    if (x < tau1) {
      xb = ws.snubar[0];
      xa = ws.alpha[0];
    } else {
      const Map1At at(ws.taunu, nr, last, x, gr);
      xb = at(ws.snubar);
      xa = at(ws.alpha);
    }
    xa = fmax(xa, 0.0);
    xb = fmax(xb, 1.0e-38);
    ws.xalpha[l] = xa;
    ws.xsbar[l] = xb;
    amax = fmax(amax, xa);
    if (l == kNx - 1) ws.last = last;
  }
  amax = g.max(amax);
  g.sync();
  const int L = ws.last;
  solve = amax > 0.0;
  if (!solve) {
    for (int l = g.r; l < kNx; l += G::N) ws.xs[l] = ws.xsbar[l];
    g.sync();
  }
  return (L > nr ? nr : L) - 1;
}

// J - S and H on the 51-point grid from XS (COEFJ.XS - XS into xw, COEFH.XS
// into xh), four interleaved partial sums per product (instruction-level
// parallelism instead of one 51-long dependent chain; the grouping differs
// from the reference's sequential sum only at rounding level), and
// KNU(1) = CK.XS in the reference order (:18700-18735)
template <class G>
__device__ __forceinline__ void josh_operators(G& g, const JoshOps& ops, const double* xs, double* xw, double* xh,
                                               double* knu1) {
  for (int l = g.r; l < kNx; l += G::N) {
    double sj[4] = {0.0, 0.0, 0.0, 0.0}, sh[4] = {0.0, 0.0, 0.0, 0.0};
    // sum k takes the terms mm = k, k+4, k+8, ... in that order
#pragma unroll 2
    for (int m0 = 0; m0 < kNx - kNx % 4; m0 += 4) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double x = xs[m0 + k];
        sj[k] = sj[k] + ops.coefj[(m0 + k) * kNx + l] * x;
        sh[k] = sh[k] + ops.coefh[(m0 + k) * kNx + l] * x;
      }
    }
#pragma unroll
    for (int k = 0; k < kNx % 4; ++k) {
      const int mm = kNx - kNx % 4 + k;
      const double x = xs[mm];
      sj[k] = sj[k] + ops.coefj[mm * kNx + l] * x;
      sh[k] = sh[k] + ops.coefh[mm * kNx + l] * x;
    }
    xw[l] = -xs[l] + ((sj[0] + sj[1]) + (sj[2] + sj[3]));
    xh[l] = (sh[0] + sh[1]) + (sh[2] + sh[3]);
  }
  if (g.r == 0) {
    double xk = 0.0;
    for (int mm = 0; mm < kNx; ++mm) xk = xk + ops.ck[mm] * xs[mm];
    *knu1 = xk;
  }
}

// ws.xs holds the solution (or XSBAR); ws.taunu, ws.rd, ws.alpha, ws.snubar
// as g_josh_prepare left them.  full (JoshWSFull or a view with the same
// members in shared memory) receives SNU, HNU, JMINS, JNU, KNU(1), MAXJ.
// hsurf_only (IFSURF = 1): only the surface flux HNU(1) is wanted; the caller
// takes it from XS where the surface is mapped, so this is the unmapped case
// (MAXJ = 1), and full needs only SNU, HNU and JMINS.  Returns the number of
// Eddington sweeps run.
template <bool hsurf_only = false, class G, class WS, class FullT>
__device__ inline int g_josh_finish(G& g, const JoshGrid& J, const JoshOps& ops, int nr, int maxj, bool mapped, WS& ws,
                                    FullT& F, const double* bnu) {
  constexpr int C = (kKwMax + G::N - 1) / G::N;
  double vj[C], vh[C];  // J - S and H of the thread's mapped depths
  if (mapped) {
    for (int l = g.r; l < kNx; l += G::N) ws.xs[l] = fmax(ws.xs[l], 1.0e-37);
    g.sync();
    if (maxj != 1) {
      josh_operators(g, ops, ws.xs, ws.xw, ws.xsbar, &F.knu1);  // XSBAR no longer needed: holds XH
      g.sync();
    }
    // XS, J - S and H back onto the depths: one bracket for the three.  J and
    // H go to memory after the sweeps, which use the same vectors below MAXJ.
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = g.r + c * G::N;
      if (j >= maxj) break;
      const double v = ws.taunu[j];
      const Map1At at(J.xtau, kNx, map1_bracket(J.xtau, kNx, v), v, J.tau());
      F.snu[j] = at(ws.xs);
      if (maxj != 1) {
        vj[c] = at(ws.xw);
        vh[c] = at(ws.xsbar);
      }
    }
    g.sync();
  }
  int sweeps = 0;
  double *snu = F.snu, *hnu = F.hnu, *jmins = F.jmins;
  if (maxj != nr) {
    const int maxj1 = (maxj == 1) ? 1 : maxj + 1;
    for (int j = maxj1 - 1 + g.r; j < nr; j += G::N) snu[j] = ws.snubar[j];
    g.sync();
    const int m = maxj - 1 > 1 ? maxj - 1 : 1;
    const int nm1 = nr - m + 1, nmj = nr - maxj + 1;
    const GridP gm{ws.rd + m - 1, nullptr}, gj{ws.rd + maxj - 1, nullptr};
    for (int l = 1; l <= 50; ++l) {
      sweeps = l;
      // negative SNU -> reset to BNU
      bool neg = false;
      for (int j = m - 1 + g.r; j < nr; j += G::N) neg |= (snu[j] <= 0.0);
      int ifneg = g.any(neg) ? 1 : 0;
      if (ifneg) {
        for (int j = m - 1 + g.r; j < nr; j += G::N) {
          ws.snubar[j] = bnu[j];
          snu[j] = bnu[j];
        }
        g.sync();
      }
      g_deriv_on(g, ws.taunu + m - 1, snu + m - 1, hnu + m - 1, nm1, gm);
      bool hneg = false;
      for (int j = m - 1 + g.r; j < nr; j += G::N) hneg |= (hnu[j] <= 0.0);
      if (g.any(hneg)) {
        ifneg = 1;
        for (int j = m - 1 + g.r; j < nr; j += G::N) {
          ws.snubar[j] = bnu[j];
          snu[j] = bnu[j];
        }
        g.sync();
        g_deriv_on(g, ws.taunu + m - 1, snu + m - 1, hnu + m - 1, nm1, gm);
      }
      for (int j = m - 1 + g.r; j < nr; j += G::N) hnu[j] = hnu[j] / 3.0;
      g.sync();
      g_deriv_on(g, ws.taunu + maxj - 1, hnu + maxj - 1, jmins + maxj - 1, nmj, gj);
      double err = 0.0;
      for (int j = maxj1 - 1 + g.r; j < nr; j += G::N) {
        if (ifneg) jmins[j] = 0.0;
        const double jv = jmins[j] + snu[j];
        if (!hsurf_only) F.jnu[j] = jv;
        const double snew = (1.0 - ws.alpha[j]) * ws.snubar[j] + ws.alpha[j] * jv;
        err += fabs(snew - snu[j]) / snew;
        snu[j] = snew;
      }
      err = g.sum(err);
      g.sync();
      if (err < 0.00001) break;
    }
  }
  if (hsurf_only) return sweeps;
  if (g.r == 0) F.maxj = maxj;
  if (maxj == 1) {
    if (g.r == 0) F.knu1 = F.jnu[0] / 3.0;
    g.sync();
    return sweeps;
  }
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int j = g.r + c * G::N;
    if (j >= maxj) break;
    jmins[j] = vj[c];
    hnu[j] = vh[c];
    snu[j] = fmax(snu[j], 1.0e-38);
    F.jnu[j] = fmax(vj[c] + snu[j], 1.0e-38);
  }
  g.sync();
  return sweeps;
}

// The whole of JOSH (IFSURF = 0) by a pair group.  ws.abtot/alpha/snubar are
// formed here from the opacity vectors; the grids are shared by the CTA.
// U: the pivot rows.  Returns the number of Eddington sweeps run.
template <class G>
__device__ inline int g_josh(G& g, const JoshGrid& J, const JoshOps& ops, int nr, const double* acont,
                             const double* aline, const double* sigmac, const double* sigmal,
                             const double* scont, const double* sline, const double* bnu, JoshWS& ws,
                             double* U, JoshWSFull& full) {
  g_josh_fill(g, nr, acont, aline, sigmac, sigmal, scont, sline, ws);
  bool mapped, solve;
  const int maxj = g_josh_prepare(g, J, nr, ws, mapped, solve);
  if (solve) solve_scatter(g, ops, ws, U);
  return g_josh_finish(g, J, ops, nr, maxj, mapped, ws, full, bnu);
}

}  // namespace atlasgpu
