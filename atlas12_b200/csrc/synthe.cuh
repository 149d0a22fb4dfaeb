// synthe.cuh -- SYNTHE hot-path kernels (sm_100a).
//
//  k_bin        line -> grid index (mod_mklinelist.f90:898-899)
//  k_continuum  continuum per depth on the grid (synthe.f90:483-516)
//  k_core       gates, line centre and Voigt core walk of every (line, depth)
//               pair (synthe.f90:559-640), one pair per lane at a time,
//               core values scattered with FP64 atomics; far-wing lines
//               recorded for k_farwing
//  k_far_*      per-(depth, tile) inverted index of the far-wing lines
//  k_farwing    the x_wing/n^2 far wings (synthe.f90:641-650) per 128-bin
//               sub-tile: distant lines as Taylor expansions about the
//               sub-tile centre, near ones bin by bin; plus the core
//               accumulator, written as the REAL(4) opacity matrix
//  k_spec_*     the wavelength loop (synthe.f90:698-718, 797-902): two
//               JOSH(1,1) solves per wavelength
#pragma once
#include "common.cuh"
#include "josh.cuh"
#include "scatter.cuh"
#include "voigt.cuh"

namespace atlasgpu {

constexpr int kTile = 1024;      // bins per far-wing tile

struct FarLine {
  int c;    // line centre nbuff (1-based)
  int n10;  // n10dop: core extent
  int m;    // maxstep: far-wing extent
  int pad;
  double x; // x_wing = profile(n10dop) * n10dop**2
};

// ---------------------------------------------------------------- binning
static __global__ void k_bin(const double* __restrict__ wl, int64_t n, double ratiolg, int ixwlbeg,
                      int32_t* __restrict__ nbuff, int64_t* __restrict__ flagged,
                      unsigned long long* __restrict__ nflag, int64_t flag_cap) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double q = log(wl[i]) / ratiolg + 0.5;
    const int ixwl = (int)q;
    nbuff[i] = ixwl - ixwlbeg + 1;
    // a 1-ulp difference in log moves q by < 1e-9: re-evaluate near-integers on the host
    if (fabs(q - rint(q)) < 1.0e-8) {
      const unsigned long long k = atomicAdd(nflag, 1ull);
      if ((int64_t)k < flag_cap) flagged[k] = i;
    }
  }
}

// ---------------------------------------------------------------- continuum
static __global__ void k_continuum(const double* __restrict__ wledge, int nedge,
                            const double* __restrict__ continall, int stride, int nrhox,
                            double wbegin, double ratio, int length, float* __restrict__ out) {
  const int j = blockIdx.y;
  const double* ab = continall + (size_t)j * stride;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < length; i += gridDim.x * blockDim.x) {
    const double w = wbegin * powi(ratio, i);
    // iedge = 1 + #{e in [2, nedge-1] : wledge(e) <= w}
    int lo = 1, hi = nedge - 1;  // answer in [1, nedge-1]
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;  // candidate iedge
      if (wledge[mid - 1] <= w) lo = mid;
      else hi = mid - 1;
    }
    const int ie = lo;
    const double wl0 = wledge[ie - 1], wl1 = wledge[ie];
    const double h = (wl0 + wl1) * 0.5;
    const double dd = powi(wl1 - wl0, 2) * 0.5;
    const double* q = ab + 3 * (ie - 1);
    const double v = ((w - h) * (w - wl1) * q[0] + (wl0 - w) * (w - wl1) * 2.0 * q[1] +
                      (w - wl0) * (w - h) * q[2]) / dd;
    float cf = (float)v;
    if (cf < -15.0f) cf = -15.0f;
    out[(size_t)j * length + i] = (float)exp10((double)cf);
  }
}

// ---------------------------------------------------------------- core pass
struct CoreArgs {
  const atlasgpu_lte_line* lines;
  int64_t n;
  int length, nrhox, nspec, maxprof, j0, nj;  // depths [j0, j0+nj)
  double resolu;
  const float* cont;     // [nrhox][length]
  const double *xnfdop, *dopple;  // [nrhox][nspec]
  const double *xne, *txnxn, *hckt;
  double* acc;           // [nrhox][length] core accumulator
  FarLine* far;          // [nj][n]
  unsigned int* nfar;    // [nj]
  // work counters (timed launches only, else null): [0] Voigt evaluations,
  // [1] far-wing bin updates the gather will make
  unsigned long long* work = nullptr;
};

// Every lane walks (line, depth) pairs on its own, one Voigt evaluation per
// trip of the loop: the centre point first, then the core points
// s = 1, 2, ... until the first value below kapmin (scattered too, as the
// reference's loop does) or s = n10dop.  The evaluation is the only
// expensive step, and all lanes with a pair run it together whatever the
// lengths of their walks, so the warp keeps its lanes supplied: it gates the
// pairs 32 at a time (a chunk of its grid-stride sequence, one pair per lane;
// the next chunk's line records are already in flight), pairs that pass both
// kapmin gates go into the warp's queue in shared memory, and when at least
// kCoreRefill lanes are idle each takes the next queued pair.  (Handing the
// candidates from lane to lane by shuffles as soon as one lane was idle took
// as many instructions as the evaluation itself.)
// With MAXPROF < n10dop the reference scatters only min(n10dop, maxstep)
// core points when no point falls below kapmin; that limit is known only
// after the walk, so such pairs walk once to decide (phase 1) and once to
// scatter (phase 2).
// A walk that reaches n10dop without a point below kapmin records its far
// wing x_wing/n^2 (n10dop < n <= maxstep) for k_farwing, through a buffer of the
// warp: the depth's list is extended 32 records at a time.  (One counter update
// per record bounded the whole kernel: all warps work on the same depth, and
// updates of one address with a returned value pass at one per ~4 clocks;
// 18.3 ms for 1M lines x 72 depths against 13.4.)
constexpr int kCoreWarps = 8;
constexpr int kCoreQueue = 64;   // fewer than 32 left over when a chunk adds up to 32
constexpr int kCoreRefill = 8;
struct CoreQueue {
  double k0[kCoreQueue], km[kCoreQueue], ad[kCoreQueue], dv[kCoreQueue];
  int nb[kCoreQueue], n10[kCoreQueue], jj[kCoreQueue];
  FarLine far[kCoreQueue];  // far-wing records not yet in their lists, pad = depth
};

// The first n (<= 32) far-wing records of a warp's buffer into their depths'
// lists, one counter update per depth (nearly always one depth); the rest moves up.
static __device__ __forceinline__ void core_flush(const CoreArgs& a, CoreQueue& Q, int lane, int n, int count) {
  constexpr unsigned FULL = 0xffffffffu;
  __syncwarp();
  FarLine f = Q.far[lane];
  const int jj = f.pad;
  unsigned todo = __ballot_sync(FULL, lane < n);
  while (todo) {
    const int lead = __ffs(todo) - 1;
    const int jl = __shfl_sync(FULL, jj, lead);
    const bool in = lane < n && jj == jl;
    const unsigned mine = __ballot_sync(FULL, in);
    unsigned base = 0;
    if (lane == lead) base = atomicAdd(a.nfar + jl, (unsigned)__popc(mine));
    base = __shfl_sync(FULL, base, lead);
    if (in) {
      f.pad = 0;
      a.far[(size_t)jj * a.n + base + __popc(mine & ((1u << lane) - 1u))] = f;
    }
    todo &= ~mine;
  }
  FarLine m = f;
  if (n + lane < count) m = Q.far[n + lane];
  __syncwarp();
  if (n + lane < count) Q.far[lane] = m;
  __syncwarp();
}

static __global__ void __launch_bounds__(32 * kCoreWarps, 4) k_core(const __grid_constant__ CoreArgs a) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ CoreQueue s_q[kCoreWarps];
  CoreQueue& Q = s_q[threadIdx.x >> 5];
  const int64_t npairs = a.n * a.nj;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int64_t pair = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * 32 + lane;  // the lane's pair of the next chunk
  unsigned long long nev = 0, nfw = 0;  // counted only when a.work is set
  // the next chunk's pair of this lane: its depth and line record, loaded one chunk ahead
  int g_j = 0;
  atlasgpu_lte_line g_line;
  g_line.nelion = 0;
  auto fetch = [&]() {
    g_line.nelion = 0;
    if (pair < npairs) {
      g_j = (int)(pair / a.n);
      g_line = a.lines[pair - (int64_t)g_j * a.n];
    }
  };
  fetch();
  int head = 0, count = 0;  // the queue, the same in every lane
  int nbuf = 0;             // buffered far-wing records
  // the lane's walk
  bool act = false;
  int phase = 0, s = 0, lim = 0, nb = 0, n10 = 0, jj = 0;
  double kappa0 = 0.0, adamp = 0.0, dv = 0.0, kapmin = 0.0;
  while (true) {
    const unsigned idle = __ballot_sync(FULL, !act);
    const int nidle = __popc(idle);
    if (nidle >= kCoreRefill) {
      // gate chunks until every idle lane can be served
      while (count < nidle && pair - lane < npairs) {
        const atlasgpu_lte_line L = g_line;
        const int jp = g_j, j = a.j0 + jp;
        pair += nw * 32;
        fetch();
        bool pass = false;
        const int nel = L.nelion - 1;
        double k0 = 0.0, km = 0.0, dp = 1.0;
        if (nel >= 0 && nel < a.nspec) {  // invalid species: no opacity
          const int ic = L.nbuff < 1 ? 1 : (L.nbuff > a.length ? a.length : L.nbuff);
          const double xd = a.xnfdop[(size_t)j * a.nspec + nel];
          dp = a.dopple[(size_t)j * a.nspec + nel];
          k0 = (double)L.cgf * xd;
          km = (double)a.cont[(size_t)j * a.length + ic - 1] * kLineCutoff;
          if (k0 >= km) {
            k0 = k0 * exp(-(double)L.elo * a.hckt[j]);
            pass = k0 >= km;
          }
        }
        const unsigned pm = __ballot_sync(FULL, pass);
        if (pass) {
          const int e = (head + count + __popc(pm & lt)) & (kCoreQueue - 1);
          Q.k0[e] = k0;
          Q.km[e] = km;
          Q.ad[e] = ((double)L.gamrf + (double)L.gamsf * a.xne[j] + (double)L.gamwf * a.txnxn[j]) / dp;
          Q.dv[e] = 1.0 / dp / a.resolu;
          Q.nb[e] = L.nbuff;
          Q.n10[e] = (int)(10.0 * dp * a.resolu);
          Q.jj[e] = jp;
        }
        count += __popc(pm);
        __syncwarp();
      }
      const int rank = __popc(idle & lt), served = min(nidle, count);
      if (!act && rank < served) {
        const int e = (head + rank) & (kCoreQueue - 1);
        act = true;
        kappa0 = Q.k0[e];
        kapmin = Q.km[e];
        adamp = Q.ad[e];
        dv = Q.dv[e];
        nb = Q.nb[e];
        n10 = Q.n10[e];
        jj = Q.jj[e];
        s = 0;
        phase = a.maxprof < n10 ? 1 : 0;
      }
      head = (head + served) & (kCoreQueue - 1);
      count -= served;
      __syncwarp();
      if (nidle == 32 && served == 0) break;
    }
    bool far = false;
    double pv = 0.0;
    if (act) {
      pv = kappa0 * voigt_weideman((double)s * dv, adamp);
      ++nev;
      double* accj = a.acc + (size_t)(a.j0 + jj) * a.length;
      if (s == 0) {
        // the line centre, then the core walk (none when n10dop < 1)
        if (nb >= 1 && nb <= a.length) atomicAdd(accj + nb - 1, pv);
        s = 1;
        act = n10 >= 1;
      } else if (phase == 1) {
        // deciding walk: the scatter limit, then the walk again from s = 1
        const bool below = pv < kapmin;
        if (below || s == n10) {
          lim = below ? s : a.maxprof;
          phase = 2;
          s = 1;
        } else {
          ++s;
        }
      } else {
        const int r = nb + s, b = nb - s;
        if (r >= 1 && r <= a.length) atomicAdd(accj + r - 1, pv);
        if (b >= 1 && b <= a.length) atomicAdd(accj + b - 1, pv);
        if (phase == 2) {
          act = s < lim;
        } else {
          act = !(pv < kapmin) && s != n10;
          far = !(pv < kapmin) && s == n10;
        }
        s += far ? 0 : 1;
      }
    }
    if (__any_sync(FULL, far)) {
      // far wing: x_wing/n**2 for n10dop < n <= maxstep
      const double xw = pv * ((double)n10 * (double)n10);
      // INT(SQRT(x_wing/kapmin))+1 capped at MAXPROF; saturate before the
      // integer conversion (the reference's INT overflows for huge ratios)
      const double q = sqrt(xw / kapmin);
      const int maxstep = q >= (double)a.maxprof ? a.maxprof : min((int)q + 1, a.maxprof);
      const int lo = max(nb - maxstep, 1), hi = min(nb + maxstep, a.length);
      const bool put = far && maxstep > n10 && lo <= hi;
      const unsigned pm = __ballot_sync(FULL, put);
      if (put) {
        FarLine f;
        f.c = nb;
        f.n10 = n10;
        f.m = maxstep;
        f.pad = jj;
        f.x = fmin(xw, 1.0e300);  // overflows REAL(4) at every n <= MAXPROF as infinity does, but 0 x is 0 (k_farwing)
        Q.far[nbuf + __popc(pm & lt)] = f;
        // bins n10 < |i - nb| <= maxstep inside the grid
        const int r0 = max(nb + n10 + 1, 1), r1 = min(nb + maxstep, a.length);
        const int b0 = max(nb - maxstep, 1), b1 = min(nb - n10 - 1, a.length);
        nfw += (unsigned long long)(r1 >= r0 ? r1 - r0 + 1 : 0) + (unsigned long long)(b1 >= b0 ? b1 - b0 + 1 : 0);
      }
      nbuf += __popc(pm);
      if (nbuf >= 32) {
        core_flush(a, Q, lane, 32, nbuf);
        nbuf -= 32;
      }
    }
  }
  if (nbuf) core_flush(a, Q, lane, nbuf, nbuf);
  if (a.work) {
    for (int o = 16; o > 0; o >>= 1) {
      nev += __shfl_xor_sync(0xffffffffu, nev, o);
      nfw += __shfl_xor_sync(0xffffffffu, nfw, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(a.work, nev);
      atomicAdd(a.work + 1, nfw);
    }
  }
}

// per depth: tile counts from the difference array, exclusive offsets
static __global__ void k_far_scan(int* __restrict__ tdiff, int ntiles, int64_t* __restrict__ off,
                           int64_t* __restrict__ fillptr, int64_t* __restrict__ total) {
  // one block per depth; sequential over tiles in chunks (ntiles is small)
  const int jj = blockIdx.x;
  if (threadIdx.x != 0) return;
  int* td = tdiff + (size_t)jj * (ntiles + 1);
  int64_t* o = off + (size_t)jj * (ntiles + 1);
  int64_t* fp = fillptr + (size_t)jj * ntiles;
  int cnt = 0;
  int64_t run = 0;
  for (int t = 0; t < ntiles; ++t) {
    cnt += td[t];
    o[t] = run;
    fp[t] = run;
    run += cnt;
  }
  o[ntiles] = run;
  total[jj] = run;
}

// The far-wing lists' counts and entries.  A block takes chunk consecutive
// far-wing records of one depth (blockIdx.y) at a time and keeps the tile
// counters in shared memory (grids with more than kFarTilesMax tiles use the global
// ones): a line touches every tile within its wing, and all lines of a depth
// touching the same few global counters bounded the fill (4.3 ms for 1M lines x
// 72 depths against 0.45 for count and fill).  chunk is kFarBlock; where that makes
// fewer blocks than the GPU has room for and the global counters are not crowded,
// kFarFew, with global counters and a warp filling a record's tiles in place of a
// thread (fill of 1,000 lines over 700 nm, 72 depths, 588 tiles: 62 us with blocks of
// 1,024, 25 with 32; over 8,818 tiles, 4 depths 622, 29; over one tile, 72 depths 10,
// 14, and of 2,000 lines 10, 20).
constexpr int kFarBlock = 1024, kFarFew = 32;
inline int far_chunk(int64_t n, int nb, int ntiles, int nsm) {
  return n * nb <= (ntiles < 512 ? 512ll : 2048ll) * nsm ? kFarFew : kFarBlock;
}
constexpr int kFarTilesMax = 8192;

__device__ __forceinline__ int2 far_tiles(const FarLine& f, int length) {
  return make_int2((max(f.c - f.m, 1) - 1) / kTile, (min(f.c + f.m, length) - 1) / kTile);
}

// op(tile, record) for every tile of the records s0 .. s1 - 1, by the whole block: a
// thread a record, or (few) a warp
template <class Op>
__device__ __forceinline__ void far_each_tile(const FarLine* __restrict__ fj, unsigned s0, unsigned s1, int length,
                                              bool few, Op&& op) {
  if (few) {
    for (unsigned s = s0 + (threadIdx.x >> 5); s < s1; s += blockDim.x >> 5) {
      const int2 t = far_tiles(fj[s], length);
      for (int q = t.x + (threadIdx.x & 31); q <= t.y; q += 32) op(q, s);
    }
  } else {
    for (unsigned s = s0 + threadIdx.x; s < s1; s += blockDim.x) {
      const int2 t = far_tiles(fj[s], length);
      for (int q = t.x; q <= t.y; ++q) op(q, s);
    }
  }
}

// tile counts of every depth as differences (tdiff zeroed before)
static __global__ void __launch_bounds__(256) k_far_count(const FarLine* __restrict__ far,
                                                          const unsigned* __restrict__ nfar, int64_t nlines,
                                                          int length, int ntiles, int chunk,
                                                          int* __restrict__ tdiff) {
  extern __shared__ int s_cnt[];
  const int jj = blockIdx.y;
  const unsigned nf = nfar[jj];
  int* td = tdiff + (size_t)jj * (ntiles + 1);
  if (blockIdx.x * chunk >= nf) return;
  const bool sm = ntiles < kFarTilesMax && chunk == kFarBlock;
  int* cnt = sm ? s_cnt : td;
  if (sm)
    for (int t = threadIdx.x; t <= ntiles; t += blockDim.x) s_cnt[t] = 0;
  __syncthreads();
  for (unsigned s0 = blockIdx.x * chunk; s0 < nf; s0 += gridDim.x * chunk)
    for (unsigned s = s0 + threadIdx.x; s < min(s0 + chunk, nf); s += blockDim.x) {
      const int2 t = far_tiles(far[(size_t)jj * nlines + s], length);
      atomicAdd(cnt + t.x, 1);
      atomicAdd(cnt + t.y + 1, -1);
    }
  __syncthreads();
  if (sm)
    for (int t = threadIdx.x; t <= ntiles; t += blockDim.x)
      if (s_cnt[t]) atomicAdd(td + t, s_cnt[t]);
}

static __global__ void __launch_bounds__(256) k_far_fill(const FarLine* __restrict__ far,
                                                         const unsigned* __restrict__ nfar, int64_t nlines,
                                                         int length, const int64_t* __restrict__ base,
                                                         int64_t* __restrict__ fillptr, int ntiles, int chunk,
                                                         int* __restrict__ csr) {
  extern __shared__ __align__(8) unsigned char s_raw[];
  int64_t* s_pos = reinterpret_cast<int64_t*>(s_raw);  // [ntiles] where the block's next entry of a tile goes
  int* s_cnt = reinterpret_cast<int*>(s_pos + ntiles);  // [ntiles] entries of the block's current records
  const int jj = blockIdx.y;
  const unsigned nf = nfar[jj];
  const FarLine* fj = far + (size_t)jj * nlines;
  unsigned long long* fp = reinterpret_cast<unsigned long long*>(fillptr) + (size_t)jj * ntiles;
  const bool few = chunk < kFarBlock, sm = ntiles < kFarTilesMax && !few;
  for (unsigned s0 = blockIdx.x * chunk; s0 < nf; s0 += gridDim.x * chunk) {
    const unsigned s1 = min(s0 + chunk, nf);
    if (sm) {
      for (int t = threadIdx.x; t < ntiles; t += blockDim.x) s_cnt[t] = 0;
      __syncthreads();
      far_each_tile(fj, s0, s1, length, few, [&](int q, unsigned) { atomicAdd(s_cnt + q, 1); });
      __syncthreads();
      for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
        if (s_cnt[t]) {
          s_pos[t] = base[jj] + (int64_t)atomicAdd(fp + t, (unsigned long long)s_cnt[t]);
          s_cnt[t] = 0;
        }
      __syncthreads();
    }
    far_each_tile(fj, s0, s1, length, few, [&](int q, unsigned s) {
      const int64_t pos = sm ? s_pos[q] + atomicAdd(s_cnt + q, 1) : base[jj] + (int64_t)atomicAdd(fp + q, 1ull);
      csr[pos] = (int)s;
    });
    __syncthreads();
  }
}

// far-wing gather + core accumulator -> REAL(4) opacity; zeroes acc for reuse.
//
// One CTA of kFarWarps warps takes one sub-tile of kSub bins at one depth, lane l
// of each warp the bins lane + 32k; its warps walk the CSR list of the kTile-bin
// tile the sub-tile belongs to in turn, 32 lines at a time (one line record per
// lane, the next group's records already in flight), and classify each line
// against the sub-tile.  Four warps where they shorten the longest lists (few
// sub-tiles, or much longer lists in the deepest layers), one where the sub-tiles
// fill the GPU by themselves and the sums of four only cost: far_four_warps.
// Measured one against four: 576 sub-tiles (0.5 nm), 500 lines 45, 22 us; 4,032 (5
// nm), 10,000 lines 166, 115; 3,072 (20 nm, 16 depths), 100,000 lines 140, 157;
// 13,824 (20 nm), 1M lines 9.7, 10.3 ms; 338,688 (700 nm), 1,000 lines 0.49, 1.63
// ms.  (With four wherever a list had fewer than 4,096 entries, up to 10,000 lines
// over 100 to 700 nm took up to 3.2 times what one warp a sub-tile takes.)
//   * distant: the whole sub-tile lies inside one far wing of the line
//     (n10 < |i - c| <= m for every bin i) and the sub-tile centre is at
//     least kFarSep bins from c.  The line's terms x/(i - c)^2 are then the
//     Taylor series in v = (i - centre)/h (h = kSub/2) about the centre,
//       x/(D + h v)^2 = sum_k (x/D^2) (k+1) (-h/D)^k v^k,  D = centre - c,
//     |h v / D| < 1/4, and the lane adds the first kFarTerms coefficients
//     (relative truncation below 1e-8).  A group of 32 whose lines are all far
//     enough away stops after 12 or 8: what is left out is below the rounding of
//     each line's own sum, since which lines share a group depends on the order
//     that the atomics gave the list;
//   * otherwise, if any of its bins is in the line's far wing, the line is
//     broadcast to the warp (shuffles) and every bin takes x * (1/n^2) itself,
//     the lines in list order.  n is a whole number, so 1/n^2 comes from a
//     table (kFarInv entries in FP64, 32 consecutive ones per load) instead of
//     a reciprocal per bin (FP32 in mixed precision, a division in FP64).
// Bounded by instruction issue, two thirds of it the direct lines (4 of a group
// of 32).  The deepest layers have the longest lists, so they are started first
// (last, they left a quarter of the chip idle at the end): 1M lines x 72 depths
// over 41,940 bins 9.1 -> 7.6 ms, 20,000 lines over 12,346 bins 0.33 -> 0.26 ms.
// At the end the lanes' and warps' coefficients are added and each bin evaluates
// the polynomial.  Most of the C3 far-wing terms come from strong lines
// thousands of bins away, so the direct work drops to a few per cent of
// the terms.
constexpr int kSub = 128;       // bins per sub-tile (one warp)
constexpr int kSubs = kTile / kSub;
constexpr int kFarSep = 256;    // minimum |centre - c| for an expansion
constexpr int kFarResident = 24;  // warps an SM holds
constexpr int kFarTerms = 16;      // Taylor terms
constexpr int kFarSep12 = 2048;    // 12 where every line of a group is this far away (|h v / D| < 1/32: 13/32^12 = 1e-17)
constexpr int kFarSep8 = 16384;    // 8 from here on (|h v / D| < 1/256: 9/256^8 = 5e-19)
constexpr int kFarInv = 65536;  // 1/n^2, n < kFarInv (512 KB)

static __global__ void k_far_inverse(double* __restrict__ inv2) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < kFarInv) inv2[n] = n ? 1.0 / ((double)n * (double)n) : 0.0;
}

// Whether four warps a sub-tile are quicker than one, in list entries that a warp
// works through (17 a us, whether few warps run or all that fit): with one the
// longest lists (maxlist: a tile's average at the depth with the most) or an even
// share of all entries, whichever is more; with four a quarter of the longest or
// the share, a fifth more for the sums, and 3 us for every round of blocks.  The
// choice is within 10 % or 5 us of the quicker one on 150 forms (0.2 to 100 nm, 1 to
// 1M lines, 16, 40 and 72 depths).
inline bool far_four_warps(double entries, double maxlist, int ntiles, int nb, int nsm) {
  const double blocks = (double)ntiles * kSubs * nb, share = entries * kSubs / ((double)kFarResident * nsm);
  const double one = share > maxlist ? share : maxlist, part = share > 0.25 * maxlist ? share : 0.25 * maxlist;
  return 1.2 * part + 8.7 * blocks / nsm < one;  // 51 entries for 5.9 blocks on every SM
}

template <int kFarWarps>
static __global__ void __launch_bounds__(32 * kFarWarps) k_farwing(const FarLine* __restrict__ far, int64_t nlines,
                                                 const int64_t* __restrict__ off,
                                                 const int64_t* __restrict__ base,
                                                 const int* __restrict__ csr, int ntiles, int length,
                                                 int j0, const double* __restrict__ inv2,
                                                 double* __restrict__ acc,
                                                 float* __restrict__ opac,
                                                 unsigned long long* __restrict__ work) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kPer = kSub / 32;
  const int jj = gridDim.y - 1 - blockIdx.y, t = blockIdx.x / kSubs, j = j0 + jj;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ double s_b[kFarWarps][kFarTerms], s_sum[kFarWarps][kSub];
  const int lo = t * kTile + (blockIdx.x % kSubs) * kSub + 1;  // first bin of the sub-tile (1-based)
  if (lo > length) return;
  const int hi = min(lo + kSub - 1, length);                   // last bin inside the grid
  const double centre = lo + 0.5 * (kSub - 1);                 // expansion centre
  const int i0 = lo + lane;                                    // bins i0 + 32k
  double sum[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) sum[k] = 0.0;
  double b[kFarTerms];
#pragma unroll
  for (int k = 0; k < kFarTerms; ++k) b[k] = 0.0;
  unsigned nexp = 0, ndir = 0;
  const int64_t* o = off + (size_t)jj * (ntiles + 1);
  const int* list = csr + base[jj] + o[t];
  const int ne = (int)(o[t + 1] - o[t]);
  if (ne == 0) {  // the core alone
    for (int i = lo + threadIdx.x; i <= hi; i += 32 * kFarWarps) {
      double& v = acc[(size_t)j * length + i - 1];
      opac[(size_t)j * length + i - 1] = (float)v;
      v = 0.0;
    }
    return;
  }
  const FarLine* fj = far + (size_t)jj * nlines;
  const FarLine none{0, 0x7fffffff, 0, 0, 0.0};  // no bin of any sub-tile in its far wing
  // two-stage prefetch: the record of the next group, the index of the one after
  constexpr int kStep = 32 * kFarWarps;
  int e = 32 * warp + lane;
  int idx = e < ne ? list[e] : -1;
  FarLine f = idx >= 0 ? fj[idx] : none;
  idx = e + kStep < ne ? list[e + kStep] : -1;
  for (int g0 = 32 * warp; g0 < ne; g0 += kStep, e += kStep) {
    const FarLine fn = idx >= 0 ? fj[idx] : none;
    idx = e + 2 * kStep < ne ? list[e + 2 * kStep] : -1;
    // distances of the nearest and the farthest bin; 0 if the centre lies inside
    const int dl = lo - f.c, dr = f.c - hi;
    const int dmin = max(max(dl, dr), 0), dmax = max(f.c - lo, hi - f.c);
    const double D = centre - (double)f.c;
    const bool distant = dmin > f.n10 && dmax <= f.m && fabs(D) >= (double)kFarSep;
    const bool direct = !distant && dmax > f.n10 && dmin <= f.m;
    if (__any_sync(FULL, distant)) {
      // 1/D from the single-precision reciprocal and one Newton-Raphson
      // step (relative error ~1e-14, far below the truncation)
      const double Ds = distant ? D : 1.0e9, x = distant ? f.x : 0.0;
      const double r0 = (double)__frcp_rn((float)Ds);
      const double r = fma(r0, fma(-Ds, r0, 1.0), r0);
      const double g = -0.5 * kSub * r, g2 = g * g, g4 = g2 * g2;
      // powers p*g^k in four independent chains (k mod 4)
      double p0 = x * r * r, p1 = p0 * g, p2 = p0 * g2, p3 = p1 * g2;
      const bool t12 = __any_sync(FULL, distant && fabs(D) < (double)kFarSep8);
      const bool t16 = __any_sync(FULL, distant && fabs(D) < (double)kFarSep12);
#pragma unroll
      for (int k = 0; k < kFarTerms; k += 4) {
        if ((k == 8 && !t12) || (k == 12 && !t16)) break;
        b[k] = fma((double)(k + 1), p0, b[k]);
        b[k + 1] = fma((double)(k + 2), p1, b[k + 1]);
        b[k + 2] = fma((double)(k + 3), p2, b[k + 2]);
        b[k + 3] = fma((double)(k + 4), p3, b[k + 3]);
        p0 *= g4;
        p1 *= g4;
        p2 *= g4;
        p3 *= g4;
      }
      nexp += distant;
    }
    // the direct lines of this group, in list order, broadcast to every bin
    unsigned bal = __ballot_sync(FULL, direct);
    ndir += __popc(bal);
    const int span = f.m - f.n10;
    while (bal) {
      const int src = __ffs(bal) - 1;
      bal &= bal - 1u;
      const int di = i0 - __shfl_sync(FULL, f.c, src);
      const int n1 = __shfl_sync(FULL, f.n10, src) + 1;
      const unsigned sp = (unsigned)__shfl_sync(FULL, span, src);
      const double x = __shfl_sync(FULL, f.x, src);
      double v[kPer];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int d = abs(di + 32 * k);
        v[k] = 0.0;
        if ((unsigned)(d - n1) < sp) v[k] = d < kFarInv ? inv2[d] : 1.0 / ((double)d * (double)d);
      }
#pragma unroll
      for (int k = 0; k < kPer; ++k) sum[k] = fma(x, v[k], sum[k]);  // x is finite
    }
    f = fn;
  }
  // the expansion: lane sums, then the warps' sums in order, then the polynomial at each bin
#pragma unroll
  for (int k = 0; k < kFarTerms; ++k) {
    for (int sh = 16; sh > 0; sh >>= 1) b[k] += __shfl_xor_sync(FULL, b[k], sh);
    if (lane == k) s_b[warp][k] = b[k];
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) s_sum[warp][lane + 32 * k] = sum[k];
  __syncthreads();
  double c[kFarTerms];
#pragma unroll
  for (int q = 0; q < kFarTerms; ++q) {
    c[q] = s_b[0][q];
#pragma unroll
    for (int w = 1; w < kFarWarps; ++w) c[q] += s_b[w][q];
  }
  double* accj = acc + (size_t)j * length;
  for (int n = threadIdx.x; n < kSub; n += 32 * kFarWarps) {
    const int i = lo + n;
    if (i > length) break;
    double near = s_sum[0][n];
#pragma unroll
    for (int w = 1; w < kFarWarps; ++w) near += s_sum[w][n];
    const double v = ((double)i - centre) * (2.0 / kSub);
    double pv = c[kFarTerms - 1];
#pragma unroll
    for (int q = kFarTerms - 2; q >= 0; --q) pv = fma(pv, v, c[q]);
    opac[(size_t)j * length + i - 1] = (float)(accj[i - 1] + (near + pv));
    accj[i - 1] = 0.0;
  }
  if (work) {
    for (int sh = 16; sh > 0; sh >>= 1) nexp += __shfl_xor_sync(FULL, nexp, sh);
    if (lane == 0) {
      atomicAdd(work + 2, (unsigned long long)nexp);
      atomicAdd(work + 3, (unsigned long long)ndir);
    }
  }
}

// ---------------------------------------------------------------- spectrum
// The wavelength loop in stages, as the RT pass: two systems per wavelength
// (the continuum alone, then with the lines), each a record in device memory.
//   k_spec_pre     warp per wavelength: the interpolated continuum, Planck
//                  terms, and for both systems INTEG and the two MAP1s onto
//                  the 51-point grid; an optically thick surface (MAXJ = 1)
//                  is finished here by its Eddington sweeps
//   k_spec_series, k_spec_solve  the scattering systems (scatter.cuh), down to
//                  H(1) = sum CH_J XS
//   k_spec_flux    flux and continuum flux of every wavelength
// One warp with the whole of JOSH and the elimination of a 51x51 matrix in
// its 30 KB of shared memory (7 warps per SM) took 3.73 ms for 12,346
// wavelengths and 12.95 ms for 41,900; the elimination of systems that a few
// series steps settle was most of it.
struct SpecWS {
  double abtot[kKwMax], alpha[kKwMax], snubar[kKwMax], taunu[kKwMax], rd[kKwMax], r2[kKwMax];
  double xsbar[kNx], xalpha[kNx], xs[kNx];
  double snu[kKwMax], hnu[kKwMax], jmins[kKwMax], bnu[kKwMax];  // the unmapped surfaces' sweeps
  double *xw, *jnu, knu1;                                      // not used with IFSURF = 1
  int last, maxj;
};
constexpr int kSpecWarps = 4;
constexpr int kSpecChunk = 32768;  // wavelengths per round: two 154-double records each, 81 MB (of 126 MB of L2)
// record: XALPHA, XSBAR, then XS (its first word becomes H(1)), the solve flag
constexpr int kSpecXs = 2 * kNx, kSpecSolve = 3 * kNx, kSpecStride = 3 * kNx + 1;
inline size_t spec_smem_bytes() { return sizeof(JoshGrid) + kSpecWarps * sizeof(SpecWS); }

struct SpecArgs {
  const JoshOps* ops;
  const double *wledge, *contabs, *contscat, *rhox, *hkt;
  int nedge, stride, nrhox, length;
  double wbegin, ratio;
  const float* opac;  // [nrhox][length]
  double *flux, *cont;
  double* rec;        // [2 * chunk][kSpecStride]: wavelength i's continuum system at 2i, total at 2i+1
  int iw0, n;         // the round's wavelengths iw0 .. iw0 + n - 1
  int per_series;     // systems per group of the series
};
__device__ __forceinline__ ScatterArgs spec_scatter_args(const SpecArgs& a) {
  ScatterArgs s{a.ops, a.rec, kSpecStride, 0, kNx, kSpecXs, kSpecSolve, 2 * a.n, a.per_series, nullptr, nullptr,
                nullptr};
  scatter_lists(s, 2 * (size_t)a.n);
  return s;
}

static __global__ void __launch_bounds__(kSpecWarps * 32, 4) k_spec_pre(SpecArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpG g(lane);
  JoshGrid& J = *reinterpret_cast<JoshGrid*>(smem_raw);
  SpecWS& S = reinterpret_cast<SpecWS*>(smem_raw + sizeof(JoshGrid))[wid];
  const int nr = a.nrhox;
  josh_grid_load(J, *a.ops, a.rhox, nr);
  if (blockIdx.x == 0 && threadIdx.x == 0) scatter_reset(spec_scatter_args(a));
  constexpr int C = (kKwMax + 31) / 32;
  for (int i = blockIdx.x * kSpecWarps + wid; i < a.n; i += gridDim.x * kSpecWarps) {
    const int iw = a.iw0 + i;
    const double wave8 = a.wbegin * powi(a.ratio, iw);
    // iedge_sv = 1 + #{e >= 2 : wledge(e) <= wave}  (setup_opacity_sv walk)
    int lo = 1, hi = a.nedge - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.wledge[mid - 1] <= wave8) lo = mid;
      else hi = mid - 1;
    }
    const int ie = lo;
    const double wl0 = a.wledge[ie - 1], wl1 = a.wledge[ie];
    const double half = (wl0 + wl1) * 0.5, del = powi(wl1 - wl0, 2) * 0.5;
    const double c1 = (wave8 - half) * (wave8 - wl1) / del;
    const double c2 = (wl0 - wave8) * (wave8 - wl1) * 2.0 / del;
    const double c3 = (wave8 - wl0) * (wave8 - half) / del;
    const double freq = kClightNms / wave8;
    const double f3 = powi(freq / 1.0e15, 3);
    double ac[C], sg[C], stim[C];
    // ACONT, SIGMAC and the source function; SNUBAR = BNU in both systems (SCONT = SLINE = BNU)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int j = lane + 32 * c;
      if (j >= nr) break;
      const double* ca = a.contabs + (size_t)j * a.stride + 3 * (ie - 1);
      const double* cs = a.contscat + (size_t)j * a.stride + 3 * (ie - 1);
      ac[c] = exp10(c1 * ca[0] + c2 * ca[1] + c3 * ca[2]);
      sg[c] = exp10(c1 * cs[0] + c2 * cs[1] + c3 * cs[2]);
      const double ehvkt = exp(-freq * a.hkt[j]);
      stim[c] = 1.0 - ehvkt;
      S.bnu[j] = kBnuPrefac * f3 * ehvkt / stim[c];
    }
    for (int sys = 0; sys < 2; ++sys) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int j = lane + 32 * c;
        if (j >= nr) break;
        // the line opacity is a REAL(4) value in the reference (ASYNTH)
        const double al = sys == 0 ? 0.0 : (double)(float)((double)a.opac[(size_t)j * a.length + iw] * stim[c]);
        const double ab = ac[c] + al + sg[c];
        S.abtot[j] = ab;
        S.alpha[j] = sg[c] / ab;
        S.snubar[j] = S.bnu[j];
      }
      g.sync();
      bool mapped, solve;
      const int maxj = g_josh_prepare(g, J, nr, S, mapped, solve);
      double* rec = a.rec + (size_t)(2 * i + sys) * kSpecStride;
      if (solve) {
        for (int l = lane; l < kNx; l += 32) {
          rec[l] = S.xalpha[l];
          rec[kNx + l] = S.xsbar[l];
        }
      } else {
        double h;
        if (mapped) {
          h = 0.0;
          for (int l = lane; l < kNx; l += 32) h += a.ops->ch[l] * fmax(S.xs[l], 1.0e-37);
          h = g.sum(h);
        } else {
          g_josh_finish<true>(g, J, *a.ops, nr, maxj, false, S, S, S.bnu);
          h = S.hnu[0];
        }
        if (lane == 0) rec[kSpecXs] = h;
      }
      if (lane == 0) rec[kSpecSolve] = solve ? 1.0 : 0.0;
      g.sync();
    }
  }
}

static __global__ void __launch_bounds__(kScatterThreads, kScatterSeriesMinBlocks) k_spec_series(SpecArgs a) {
  scatter_series_body<true>(spec_scatter_args(a));
}
static __global__ void __launch_bounds__(kScatterThreads, kScatterSolveMinBlocks) k_spec_solve(SpecArgs a) {
  scatter_solve_body<true>(spec_scatter_args(a));
}

// resid * continuum, as the reference writes the flux (synthe.f90:712-718)
static __global__ void k_spec_flux(SpecArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double* rec = a.rec + (size_t)(2 * i) * kSpecStride;
  const double surf = rec[kSpecXs], hnu = rec[kSpecStride + kSpecXs];
  a.flux[a.iw0 + i] = hnu / surf * surf;
  a.cont[a.iw0 + i] = surf;
}

// ---------------------------------------------------------------- NLTE list
// compute_line_opacity's normal-metal branch (TYPE 0, 3 and the He I
// fallthrough TYPE <= -3; synthe_module.f90:3400-3458), its autoionizing (Shore)
// lines (:3609-3650) and merged-continuum edges (:3652-3696), FP64.  The wings
// of a (record, depth) are walked over consecutive grid points, one per lane;
// the first lane below the cutoff ends a wing (metals, red: tested before the
// add; everywhere else after it).  Points blueward of WCON are skipped,
// WCON..WTAIL tapers.  Grid wavelengths are wbegin * ratio**(i-1) (the reference
// walks them by repeated multiplication; the two agree to ~1e-11 relative).
//
// Most wings end within a few steps of 32 points, a Shore line's or an edge's
// run over the window (15,000 points for 12 nm at 390 nm), and those few chains
// of 470 latency-bound steps were the kernel.  So a warp walks a wing for some
// steps and then lists what is left; a block per listed wing walks on, 256 points
// a step (k_synthe_nlte_rest).  With the wavelengths from a table (a power per
// point before) and one division a Shore point for five: 300 records, 72 depths,
// 12 nm: 818 -> 290 us.
// A block takes 256 lanes for what is often a part of that, and the set-up again,
// so listing only pays for a chip that is not full or a chain that is long: after
// 8 steps where a resident warp has two (record, depth) pairs at most (30 records,
// 72 depths, 4 nm at 400 nm: 152 us with one warp a wing and powers, 120 after 64
// steps, 58 after 8), after 64 steps otherwise (3,000 records, 1 nm at 900 nm: 497,
// 382, 655; 300 records, 12 nm: 577, 272, 258), never in a window of up to
// kNlteShort points (1,000 records, half of them Shore, 1 nm at 900 nm: 243, 183,
// 372).
struct NlteRest {
  int64_t pair;  // record * nrhox + depth
  int pos, red;  // next grid point (1-based) and direction
};
constexpr int kNlteSoloFew = 8, kNlteSolo = 64;  // steps of a warp before a wing is listed
constexpr int kNlteResident = 24;                // warps an SM holds
constexpr int kNlteWarps = 8;               // warps per listed wing
constexpr int64_t kNlteRestMax = 1 << 18;   // a full list: the warp walks its wing to the end
struct NlteArgs {
  const atlasgpu_nlte_line* rec;
  int64_t n;
  int length, nrhox, nspec;
  double wbegin, ratio, wlend, dopratio;
  const double *wave, *freq;        // [length] grid wavelengths and frequencies (k_grid_wave)
  const float* cont;                // [nrhox][length]
  const double *xnfdop, *dopple;    // [nrhox][nspec]
  const double *xne, *txnxn, *hckt, *emerge;  // [nrhox]
  const double* contx;              // CONTX(26,17) column-major
  double* acc;                      // [nrhox][length]
  NlteRest* rest;                   // [restcap]
  int* nrest;                       // items listed, items taken (2 words)
  int restcap, solo;                // wings the list holds, steps before a wing is listed
  const double* xnfpel = nullptr;   // [nrhox][nspec] XNFPEL = populations / RHO; null: Shore lines skipped
  // merged-continuum edges (TYPE >= 4): per record its ordinal m (-1: none)
  // and per (m, depth) the grid indices NBUFF1, NBUFF2, NBUFF3 and a flag
  // (0: the edge misses the grid), computed on the host with the C library
  const int* mord = nullptr;
  const int4* mbins = nullptr;
};

// (and the unit-19 list's counters, if there is one, zeroed)
static __global__ void k_grid_wave(double wbegin, double ratio, int length, double* __restrict__ wave,
                                   double* __restrict__ freq, int* __restrict__ nrest) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (nrest && i < 2) nrest[i] = 0;
  if (i >= length) return;
  const double w = wbegin * powi(ratio, i);
  wave[i] = w;
  freq[i] = kClightNms / w;
}

// one (record, depth): what its points need, and where its wings start
struct NlteWalk {
  int kind;  // 0 metal, 1 Shore, 2 merged-continuum edge
  double k0, wl, wcon, wtail, rtaper, adamp, rdopwl;  // metal (k0, wl: all)
  double frelin, gr2, gs, gw;                         // Shore: GAMMAS, GAMMAW, 2 / GAMMAR
  int flat, last;                                     // edge: flat to here, zero at
  int red, redend, blue;                              // first points (0: no such wing), last red point
};

__device__ __forceinline__ bool nlte_setup(const NlteArgs& a, int64_t p, NlteWalk& w) {
  const int64_t il = p / a.nrhox;
  const int j = (int)(p - il * a.nrhox);
  const atlasgpu_nlte_line r = a.rec[il];
  const int t = r.itype;
  w.red = w.blue = 0;
  w.redend = a.length;
  if (t >= 4) {
    // flat to NBUFF2, then tapering to zero at NBUFF3
    if (!a.mbins) return false;
    const int m = a.mord[il];
    if (m < 0) return false;
    const int4 b = a.mbins[(size_t)m * a.nrhox + j];
    if (!b.w) return false;
    w.kind = 2;
    w.k0 = (double)r.gf * a.xnfpel[(size_t)j * a.nspec + r.nelion - 1] * exp(-(double)r.elo * a.hckt[j]);
    w.rtaper = 1.0 / (double)(b.z - b.y);
    w.flat = b.y;
    w.last = b.z;
    w.red = b.x;
    w.redend = b.z < a.length ? b.z : a.length;
    return true;
  }
  const bool shore = t == 1 && a.xnfpel;
  if (!(shore || t == 0 || t == 3 || t <= -3) || r.nelion < 1 || r.nelion > a.nspec) return false;
  const float* cont = a.cont + (size_t)j * a.length;
  const int nbuff = r.nbuff, nel = r.nelion - 1;
  const int ic = nbuff < 1 ? 1 : (nbuff > a.length ? a.length : nbuff);
  const double kapmin = (double)cont[ic - 1] * kLineCutoff;
  w.wl = r.wlvac * a.dopratio;
  if (shore) {
    // KAPPA0 = GAMMAW*GF*XNFPEL with the two continuum gates around the Boltzmann
    // factor, then the Fano profile KAPPA0*(GAMMAS*EPSIL + GAMMAW)/(EPSIL**2+1)/GAMMAW,
    // EPSIL = 2*(FREQ - FRELIN)/GAMMAR
    w.kind = 1;
    w.gs = (double)r.gammas;
    w.gw = (double)r.gammaw;
    w.gr2 = 2.0 / (double)r.gammar;
    double kappa0 = w.gw * (double)r.gf * a.xnfpel[(size_t)j * a.nspec + nel];
    if (kappa0 < kapmin) return false;
    kappa0 = kappa0 * exp(-(double)r.elo * a.hckt[j]);
    if (kappa0 < kapmin) return false;
    w.k0 = kappa0 / w.gw;
    w.frelin = kClightNms / w.wl;
  } else {
    const double xd = a.xnfdop[(size_t)j * a.nspec + nel], dp = a.dopple[(size_t)j * a.nspec + nel];
    double kappa0 = (double)r.gf * xd;
    if (kappa0 < kapmin) return false;
    kappa0 = kappa0 * exp(-(double)r.elo * a.hckt[j]);
    if (kappa0 < kapmin) return false;
    w.kind = 0;
    w.k0 = kappa0;
    w.wcon = w.wtail = 0.0;
    if (r.ncon > 0) {
      const double cx = a.contx[(size_t)(r.nelionx - 1) * 26 + (r.ncon - 1)];
      w.wcon = 1.0e7 / (cx - a.emerge[j]) * a.dopratio;
      w.wtail = 1.0e7 / (cx - a.emerge[j] - 500.0) * a.dopratio;
    }
    w.rtaper = 1.0 / (w.wtail - w.wcon);
    w.adamp = ((double)r.gammar + (double)r.gammas * a.xne[j] + (double)r.gammaw * a.txnxn[j]) / dp;
    w.rdopwl = 1.0 / (dp * w.wl);
  }
  bool blue = true;
  if (w.wl <= a.wlend) {
    w.red = nbuff > 1 ? nbuff : 1;
    blue = !((shore ? nbuff : w.red) == 1 || w.wl < a.wbegin);
  }
  if (blue) w.blue = (a.length + 1 < nbuff ? a.length + 1 : nbuff) - 1;
  return true;
}

// walks one wing from point pos on, 32 (kBlock: 32 kNlteWarps) points a step;
// returns where it stands after maxsteps steps, 0 when the wing has ended
template <bool kBlock>
__device__ __forceinline__ int nlte_walk(const NlteArgs& a, const double* waves, const double* freqs,
                                         const NlteWalk& w, int j, bool red, int pos, int maxsteps, int t,
                                         BlockVote<kNlteWarps>* vote, int& par) {
  constexpr int W = kBlock ? 32 * kNlteWarps : 32;
  const float* cont = a.cont + (size_t)j * a.length;
  double* acc = a.acc + (size_t)j * a.length;
  const bool before = w.kind == 0 && red;  // tested before the add
  for (int steps = 0; red ? pos <= w.redend : pos >= 1; pos += red ? W : -W) {
    if (steps++ == maxsteps) return pos;
    const int ib = red ? pos + t : pos - t;
    bool use = red ? ib <= w.redend : ib >= 1, stop = false;
    double kappa = 0.0;
    if (use) {
      if (w.kind == 0) {
        const double wave = waves[ib - 1];
        use = wave >= w.wcon;
        if (use) {
          kappa = w.k0 * voigt_weideman(fabs(wave - w.wl) * w.rdopwl, w.adamp);
          if (wave < w.wtail) kappa = kappa * ((wave - w.wcon) * w.rtaper);
          stop = kappa < (double)cont[ib - 1] * kLineCutoff;
        }
      } else if (w.kind == 1) {
        const double eps = w.gr2 * (freqs[ib - 1] - w.frelin);
        kappa = w.k0 * (w.gs * eps + w.gw) / (eps * eps + 1.0);
        stop = kappa < (double)cont[ib - 1] * kLineCutoff;
      } else {
        kappa = ib > w.flat ? w.k0 * ((double)(w.last - ib) * w.rtaper) : w.k0;
      }
    }
    int first, none;
    if (kBlock) {
      block_vote(*vote, par, stop, false, t, first, none);
    } else {
      const unsigned sb = __ballot_sync(0xffffffffu, stop);
      first = sb ? __ffs(sb) - 1 : 32;
    }
    if (use && (before ? t < first : t <= first)) atomicAdd(acc + ib - 1, kappa);
    if (first < W) return 0;
  }
  return 0;
}

// kShort: a window of at most kNlteShort points.  A warp walks its wings to their
// ends, nothing is listed, and the wavelengths (the same ones) are formed by every
// block in shared memory: one launch in place of three (50 points, 5 records, 16
// depths, the call: 94 us with three launches and a memset, 84 with one).
constexpr int kNlteShort = 1024;
static_assert(kNlteShort <= 32 * kNlteSolo, "a wing of a short window is never listed");
template <bool kShort>
static __global__ void __launch_bounds__(256) k_synthe_nlte(const __grid_constant__ NlteArgs a) {
  __shared__ double s_wave[kShort ? kNlteShort : 1], s_freq[kShort ? kNlteShort : 1];
  if (kShort) {
    for (int i = threadIdx.x; i < a.length; i += blockDim.x) {
      const double w = a.wbegin * powi(a.ratio, i);
      s_wave[i] = w;
      s_freq[i] = kClightNms / w;
    }
    __syncthreads();
  }
  const double *waves = kShort ? s_wave : a.wave, *freqs = kShort ? s_freq : a.freq;
  const int lane = threadIdx.x & 31;
  const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t npair = a.n * a.nrhox;
  int par = 0;
  for (int64_t p = w0; p < npair; p += nw) {
    NlteWalk w;
    if (!nlte_setup(a, p, w)) continue;
    const int j = (int)(p % a.nrhox);
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      const bool red = dir == 0;
      int pos = red ? w.red : w.blue;
      if (pos < 1) continue;
      pos = nlte_walk<false>(a, waves, freqs, w, j, red, pos, kShort ? kNlteSolo : a.solo, lane, nullptr, par);
      if (kShort || pos < 1) continue;
      int slot = 0;
      if (lane == 0) slot = atomicAdd(a.nrest, 1);
      slot = __shfl_sync(0xffffffffu, slot, 0);
      if (slot < a.restcap) {
        if (lane == 0) a.rest[slot] = NlteRest{p, pos, red};
      } else {
        nlte_walk<false>(a, waves, freqs, w, j, red, pos, 0x7fffffff, lane, nullptr, par);
      }
    }
  }
}

// (items are taken from the list in turn: their lengths differ by factors of ten)
static __global__ void __launch_bounds__(32 * kNlteWarps, 3) k_synthe_nlte_rest(const __grid_constant__ NlteArgs a) {
  __shared__ BlockVote<kNlteWarps> vote;
  __shared__ NlteWalk walk;
  __shared__ NlteRest item;
  __shared__ int s_i;
  const int n = min(a.nrest[0], a.restcap);
  int par = 0;
  for (;;) {
    if (threadIdx.x < 32) {
      int i = 0;
      if (threadIdx.x == 0) i = atomicAdd(a.nrest + 1, 1);
      i = __shfl_sync(0xffffffffu, i, 0);
      NlteWalk w;
      NlteRest q{0, 0, 0};
      if (i < n) {
        q = a.rest[i];
        nlte_setup(a, q.pair, w);
      }
      if (threadIdx.x == 0) {
        s_i = i;
        if (i < n) {
          walk = w;
          item = q;
        }
      }
    }
    __syncthreads();
    if (s_i >= n) break;
    const NlteWalk w = walk;
    const NlteRest q = item;
    nlte_walk<true>(a, a.wave, a.freq, w, (int)(q.pair % a.nrhox), q.red != 0, q.pos, 0x7fffffff, threadIdx.x, &vote,
                    par);
    __syncthreads();
  }
}

// opacity [nrhox][length] (REAL(4)) += the FP64 contribution
static __global__ void k_add_f64_to_f32(const double* __restrict__ acc, float* __restrict__ out, int64_t n) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    out[e] = (float)((double)out[e] + acc[e]);
}

}  // namespace atlasgpu
