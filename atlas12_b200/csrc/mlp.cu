// mlp.cu -- the learned warm start's network: a dense tanh MLP
// (nin -> nh1 -> nh2 -> nout, FP32 weights) with hand-written forward,
// backward and Adam kernels.  It maps stellar parameters to a starting
// structure; the unmodified ATLAS12 iteration still judges convergence, so
// the network only shortens the iteration.  No reference counterpart (the
// reference starts from a tabulated model).
//
// Layers: h1 = tanh(W1 x + b1), h2 = tanh(W2 h1 + b2), y = W3 h2 + b3,
// W_l stored [out][in] row-major.  Loss: mean over samples and outputs of
// (y - target)^2.  Every sum runs in a fixed order (chunk by chunk, then folds of
// K groups and of per-block partials in fixed orders), so results repeat exactly.
//
// A training batch is 64 samples: each of the eight products is 4 MFLOP, and
// the time is latency and launches.  With 32x32 tiles, one 32-deep chunk in
// flight and 16 blocks a product took 14 us; 16x16 tiles (64 to 256 blocks), K
// split over four groups of a block and the next chunk's loads in flight
// before a chunk is multiplied take 6 us.  The bias gradients are row sums of tiles that
// the weight gradients load anyway, the loss and its gradient are the last
// layer's epilogue, and a layer's two backward products share a launch: 13
// launches a step became 6.  From nsm tiles of 64x64 on the product is bound by
// arithmetic and takes those (4x4 per thread).  Loss and gradient plus a forward
// pass of 64 samples: kernels 176 -> 52 us; 4,000 samples 1860 -> 457 us.
#include <cmath>
#include <vector>

#include "api_common.cuh"

using namespace atlasgpu;

struct atlasgpu_mlp {
  int nin, nh1, nh2, nout;
  int64_t nparam;
  float *w, *g, *m, *v;   // parameters, gradient, Adam moments [nparam]
  int64_t step = 0;
  // activations / gradients for up to cap samples
  int cap = 0;
  float *x, *t, *h1, *h2, *y, *d1, *d2, *dy, *lpart;
  float* loss;       // [1]
  unsigned* ticket;  // [1] blocks of the last layer that are done (0 between launches)
};

namespace {

// One product C[m][n] = sum_k A(m,k) B(k,n) with A(m,k) = A[m*sam + k*sak],
// B(k,n) = B[k*sbk + n*sbn] (one stride of each is 1), and what its epilogue does.
struct Prod {
  int M, N, K;
  const float* A;
  int sam, sak;
  const float* B;
  int sbk, sbn;
  float* C;           // [M][N]
  const float* bias;  // + bias[n], or null
  int act;            // then tanh
  const float* pact;  // result * (1 - pact(m,n)^2): tanh derivative of a layer output [M][N], or null
  float* rowsum;      // [M] sum_k A(m,k), or null
  // the last layer's loss: dy = 2 (y - t) / (M N) and sum of (y - t)^2 / (M N), or null
  const float* t;
  float *dy, *part, *loss;
  unsigned* ticket;
};
struct Prods {
  Prod p[2];
  int tiles0;  // blocks of p[0]; the rest are p[1]'s
};

constexpr int kMlpThreads = 256;

__device__ __forceinline__ float block_sum(float v, float* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = kMlpThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  const float r = sh[0];
  __syncthreads();
  return r;
}

// BM x BN tiles, chunks of BK, TM x TN outputs a thread, KG groups of the block
// taking every KG-th chunk; the next chunk's loads are issued before a chunk is
// multiplied
template <int BM, int BN, int BK, int TM, int TN, int KG>
__global__ void __launch_bounds__(kMlpThreads) k_prod(const __grid_constant__ Prods ps) {
  constexpr int GT = kMlpThreads / KG;  // threads of a group
  static_assert((BM / TM) * (BN / TN) == GT && KG * BM * BN >= kMlpThreads, "tile shape");
  constexpr int LA = BM * BK / GT, LB = BN * BK / GT;
  __shared__ float As[KG][BK][BM + 1], Bs[KG][BK][BN + 1];
  __shared__ float red[KG > 1 ? KG * BM * BN : kMlpThreads];
  const bool second = (int)blockIdx.x >= ps.tiles0;
  const Prod& p = ps.p[second];
  const int tile = blockIdx.x - (second ? ps.tiles0 : 0), ntn = (p.N + BN - 1) / BN;
  const int m0 = tile / ntn * BM, n0 = tile % ntn * BN;
  const int g = threadIdx.x / GT, t = threadIdx.x % GT;
  const int tx = t % (BN / TN), ty = t / (BN / TN);
  float ra[LA], rb[LB], acc[TM][TN] = {}, rs[TM] = {};
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < LA; ++q) {
      const int e = q * GT + t;
      const int k = p.sak == 1 ? e % BK : e / BM, m = p.sak == 1 ? e / BK : e % BM;
      ra[q] = (m0 + m < p.M && k0 + k < p.K) ? p.A[(size_t)(m0 + m) * p.sam + (size_t)(k0 + k) * p.sak] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < LB; ++q) {
      const int e = q * GT + t;
      const int k = p.sbk == 1 ? e % BK : e / BN, n = p.sbk == 1 ? e / BK : e % BN;
      rb[q] = (n0 + n < p.N && k0 + k < p.K) ? p.B[(size_t)(k0 + k) * p.sbk + (size_t)(n0 + n) * p.sbn] : 0.f;
    }
  };
  const bool rows = p.rowsum && n0 == 0 && tx == 0;
  fetch(g * BK);
  for (int c = 0; c * KG * BK < p.K; ++c) {
#pragma unroll
    for (int q = 0; q < LA; ++q) {
      const int e = q * GT + t;
      As[g][p.sak == 1 ? e % BK : e / BM][p.sak == 1 ? e / BK : e % BM] = ra[q];
    }
#pragma unroll
    for (int q = 0; q < LB; ++q) {
      const int e = q * GT + t;
      Bs[g][p.sbk == 1 ? e % BK : e / BN][p.sbk == 1 ? e / BK : e % BN] = rb[q];
    }
    __syncthreads();
    if ((c + 1) * KG * BK < p.K) fetch(((c + 1) * KG + g) * BK);
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[g][k][ty * TM + i];
#pragma unroll
      for (int i = 0; i < TN; ++i) b[i] = Bs[g][k][tx * TN + i];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int l = 0; l < TN; ++l) acc[i][l] = fmaf(a[i], b[l], acc[i][l]);
      if (rows)
#pragma unroll
        for (int i = 0; i < TM; ++i) rs[i] += a[i];
    }
    __syncthreads();
  }
  const float scale = 1.f / ((float)p.M * (float)p.N);
  float lsum = 0.f;
  auto finish = [&](int m, int n, float v) {
    if (m >= p.M || n >= p.N) return;
    const size_t e = (size_t)m * p.N + n;
    if (p.bias) v += p.bias[n];
    if (p.act) v = tanhf(v);
    if (p.pact) v = v * (1.f - p.pact[e] * p.pact[e]);
    p.C[e] = v;
    if (p.dy) {
      const float d = v - p.t[e];
      p.dy[e] = 2.f * d * scale;
      lsum += d * d;
    }
  };
  if (KG > 1) {
    __shared__ float rrow[KG][BM];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int l = 0; l < TN; ++l) red[(g * BM + ty * TM + i) * BN + tx * TN + l] = acc[i][l];
    if (rows)
#pragma unroll
      for (int i = 0; i < TM; ++i) rrow[g][ty * TM + i] = rs[i];
    __syncthreads();
    for (int e = threadIdx.x; e < BM * BN; e += kMlpThreads) {
      float v = red[e];
#pragma unroll
      for (int q = 1; q < KG; ++q) v += red[q * BM * BN + e];
      finish(m0 + e / BN, n0 + e % BN, v);
    }
    if (p.rowsum && n0 == 0 && threadIdx.x < BM && m0 + threadIdx.x < p.M) {
      float v = rrow[0][threadIdx.x];
#pragma unroll
      for (int q = 1; q < KG; ++q) v += rrow[q][threadIdx.x];
      p.rowsum[m0 + threadIdx.x] = v;
    }
  } else {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int l = 0; l < TN; ++l) finish(m0 + ty * TM + i, n0 + tx * TN + l, acc[i][l]);
    if (rows)
#pragma unroll
      for (int i = 0; i < TM; ++i)
        if (m0 + ty * TM + i < p.M) p.rowsum[m0 + ty * TM + i] = rs[i];
  }
  if (!p.dy) return;
  // the loss: per-block partials, summed in a fixed order by the last block
  __syncthreads();
  lsum = block_sum(lsum, red);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    p.part[tile] = lsum;
    __threadfence();
    last = atomicAdd(p.ticket, 1u) == (unsigned)ps.tiles0 - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  float v = 0.f;
  for (int i = threadIdx.x; i < ps.tiles0; i += kMlpThreads) v += __ldcg(p.part + i);
  v = block_sum(v, red);
  if (threadIdx.x == 0) {
    *p.loss = v * scale;
    *p.ticket = 0;
  }
}

__global__ void k_adam(int64_t n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// gather rows idx[0..n) of src [*][w] into dst [n][w]
__global__ void k_gather(int n, int w, const int* __restrict__ idx, const float* __restrict__ src,
                         float* __restrict__ dst) {
  const int64_t total = (int64_t)n * w;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(e / w), c = (int)(e % w);
    dst[e] = src[(size_t)idx[r] * w + c];
  }
}

struct Off {
  int64_t w1, b1, w2, b2, w3, b3;
};
Off offsets(const atlasgpu_mlp* p) {
  Off o;
  o.w1 = 0;
  o.b1 = o.w1 + (int64_t)p->nh1 * p->nin;
  o.w2 = o.b1 + p->nh1;
  o.b2 = o.w2 + (int64_t)p->nh2 * p->nh1;
  o.w3 = o.b2 + p->nh2;
  o.b3 = o.w3 + (int64_t)p->nout * p->nh2;
  return o;
}

constexpr int kSmallTile = 16, kLargeTile = 64;
int tiles(const Prod& p, int edge) { return ((p.M + edge - 1) / edge) * ((p.N + edge - 1) / edge); }

// one or two independent products: together in small tiles, each by itself in
// large ones where those fill the chip
int products(atlasgpu_ctx* ctx, const Prod& a, const Prod* b) {
  const bool la = tiles(a, kLargeTile) >= ctx->nsm, lb = b && tiles(*b, kLargeTile) >= ctx->nsm;
  if (b && (la || lb)) {
    const int r = products(ctx, a, nullptr);
    return r ? r : products(ctx, *b, nullptr);
  }
  Prods ps{{a, b ? *b : a}, tiles(a, la ? kLargeTile : kSmallTile)};
  const int blocks = ps.tiles0 + (b ? tiles(*b, kSmallTile) : 0);
  if (la) k_prod<kLargeTile, kLargeTile, 16, 4, 4, 1><<<blocks, kMlpThreads, 0, ctx->stream>>>(ps);
  else k_prod<kSmallTile, kSmallTile, 32, 2, 2, 4><<<blocks, kMlpThreads, 0, ctx->stream>>>(ps);
  CKL(ctx);
  return 0;
}

int ensure_cap(atlasgpu_ctx* ctx, atlasgpu_mlp* p, int n) {
  if (n <= p->cap) return 0;
  float** bufs[] = {&p->x, &p->t, &p->h1, &p->h2, &p->y, &p->d1, &p->d2, &p->dy, &p->lpart};
  p->cap = 0;
  for (float** b : bufs) {
    if (*b) cudaFree(*b);
    *b = nullptr;
  }
  Prod last{};
  last.M = n;
  last.N = p->nout;
  const size_t counts[] = {(size_t)n * p->nin, (size_t)n * p->nout, (size_t)n * p->nh1, (size_t)n * p->nh2,
                           (size_t)n * p->nout, (size_t)n * p->nh1, (size_t)n * p->nh2, (size_t)n * p->nout,
                           (size_t)tiles(last, kSmallTile)};
  for (int i = 0; i < 9; ++i)
    if (cudaMalloc(bufs[i], sizeof(float) * counts[i]) != cudaSuccess) {
      cudaGetLastError();
      return fail(ctx, ATLASGPU_ENOMEM, "mlp: activations for %d samples", n);
    }
  p->cap = n;
  return 0;
}

// y = act(x W^T + b) of one layer
Prod layer(int n, int nin, int nout, const float* x, const float* w, const float* b, int act, float* y) {
  Prod p{};
  p.M = n, p.N = nout, p.K = nin;
  p.A = x, p.sam = nin, p.sak = 1;
  p.B = w, p.sbk = 1, p.sbn = nin;
  p.bias = b, p.act = act, p.C = y;
  return p;
}
// dW = d^T h and db = column sums of d
Prod grad_w(int n, int nin, int nout, const float* d, const float* h, float* gw, float* gb) {
  Prod p{};
  p.M = nout, p.N = nin, p.K = n;
  p.A = d, p.sam = 1, p.sak = nout;
  p.B = h, p.sbk = nin, p.sbn = 1;
  p.C = gw, p.rowsum = gb;
  return p;
}
// d of the layer below: (d W) (1 - h^2)
Prod grad_x(int n, int nin, int nout, const float* d, const float* w, const float* h, float* dx) {
  Prod p{};
  p.M = n, p.N = nin, p.K = nout;
  p.A = d, p.sam = nout, p.sak = 1;
  p.B = w, p.sbk = nin, p.sbn = 1;
  p.pact = h, p.C = dx;
  return p;
}

// forward over n samples already in p->x; with d_loss also the loss over p->t and its gradient in p->dy
int forward(atlasgpu_ctx* ctx, atlasgpu_mlp* p, int n, float* d_loss = nullptr) {
  const Off o = offsets(p);
  int r;
  if ((r = products(ctx, layer(n, p->nin, p->nh1, p->x, p->w + o.w1, p->w + o.b1, 1, p->h1), nullptr)) ||
      (r = products(ctx, layer(n, p->nh1, p->nh2, p->h1, p->w + o.w2, p->w + o.b2, 1, p->h2), nullptr)))
    return r;
  Prod last = layer(n, p->nh2, p->nout, p->h2, p->w + o.w3, p->w + o.b3, 0, p->y);
  if (d_loss) last.t = p->t, last.dy = p->dy, last.part = p->lpart, last.loss = d_loss, last.ticket = p->ticket;
  return products(ctx, last, nullptr);
}

// gradient (p->g) from p->dy and the activations of forward
int backward(atlasgpu_ctx* ctx, atlasgpu_mlp* p, int n) {
  const Off o = offsets(p);
  int r;
  const Prod x2 = grad_x(n, p->nh2, p->nout, p->dy, p->w + o.w3, p->h2, p->d2);
  const Prod x1 = grad_x(n, p->nh1, p->nh2, p->d2, p->w + o.w2, p->h1, p->d1);
  if ((r = products(ctx, grad_w(n, p->nh2, p->nout, p->dy, p->h2, p->g + o.w3, p->g + o.b3), &x2)) ||
      (r = products(ctx, grad_w(n, p->nh1, p->nh2, p->d2, p->h1, p->g + o.w2, p->g + o.b2), &x1)))
    return r;
  return products(ctx, grad_w(n, p->nin, p->nh1, p->d1, p->x, p->g + o.w1, p->g + o.b1), nullptr);
}

// splitmix64 for the initial weights (deterministic per seed)
uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

extern "C" {

int atlasgpu_mlp_create(atlasgpu_ctx* ctx, int nin, int nh1, int nh2, int nout, uint64_t seed,
                        atlasgpu_mlp** out) {
  if (!ctx || !out || nin < 1 || nh1 < 1 || nh2 < 1 || nout < 1)
    return fail(ctx, ATLASGPU_EINVAL, "mlp_create: bad shape");
  *out = nullptr;
  cudaSetDevice(ctx->device);
  auto* p = new atlasgpu_mlp();
  p->nin = nin;
  p->nh1 = nh1;
  p->nh2 = nh2;
  p->nout = nout;
  const Off o = offsets(p);
  p->nparam = o.b3 + nout;
  float** bufs[] = {&p->w, &p->g, &p->m, &p->v};
  for (float** b : bufs)
    if (cudaMalloc(b, sizeof(float) * p->nparam) != cudaSuccess) {
      delete p;
      return fail(ctx, ATLASGPU_ENOMEM, "mlp_create");
    }
  if (cudaMalloc(&p->loss, sizeof(float)) != cudaSuccess || cudaMalloc(&p->ticket, sizeof(unsigned)) != cudaSuccess) {
    delete p;
    return fail(ctx, ATLASGPU_ENOMEM, "mlp_create");
  }
  // Glorot-uniform weights, zero biases
  std::vector<float> h(p->nparam, 0.f);
  uint64_t s = seed;
  auto fill = [&](int64_t off, int fan_out, int fan_in) {
    const double lim = std::sqrt(6.0 / (fan_in + fan_out));
    for (int64_t i = 0; i < (int64_t)fan_out * fan_in; ++i) {
      const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
      h[off + i] = (float)((2.0 * u - 1.0) * lim);
    }
  };
  fill(o.w1, nh1, nin);
  fill(o.w2, nh2, nh1);
  fill(o.w3, nout, nh2);
  // on the context's stream, as all that reads them (a non-blocking stream does not wait for the default one)
  cudaStream_t st = ctx->stream;
  const size_t bytes = sizeof(float) * p->nparam;
  cudaError_t e = cudaMemcpyAsync(p->w, h.data(), bytes, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(p->m, 0, bytes, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(p->v, 0, bytes, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(p->ticket, 0, sizeof(unsigned), st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    atlasgpu_mlp_destroy(ctx, p);
    return fail(ctx, ATLASGPU_ECUDA, "mlp_create: %s", cudaGetErrorString(e));
  }
  *out = p;
  return 0;
}

int atlasgpu_mlp_destroy(atlasgpu_ctx* ctx, atlasgpu_mlp* p) {
  if (!p) return ATLASGPU_EINVAL;
  if (ctx) {
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
  }
  float* bufs[] = {p->w, p->g, p->m, p->v, p->x, p->t, p->h1, p->h2, p->y, p->d1, p->d2, p->dy, p->lpart, p->loss};
  for (float* b : bufs)
    if (b) cudaFree(b);
  if (p->ticket) cudaFree(p->ticket);
  delete p;
  return 0;
}

int64_t atlasgpu_mlp_nparam(atlasgpu_mlp* p) { return p ? p->nparam : -1; }

int atlasgpu_mlp_get_params(atlasgpu_ctx* ctx, atlasgpu_mlp* p, float* out) {
  if (!ctx || !p || !out) return fail(ctx, ATLASGPU_EINVAL, "mlp_get_params");
  cudaSetDevice(ctx->device);
  CK(cudaMemcpyAsync(out, p->w, sizeof(float) * p->nparam, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return 0;
}

int atlasgpu_mlp_set_params(atlasgpu_ctx* ctx, atlasgpu_mlp* p, const float* in) {
  if (!ctx || !p || !in) return fail(ctx, ATLASGPU_EINVAL, "mlp_set_params");
  cudaSetDevice(ctx->device);
  CK(cudaMemcpyAsync(p->w, in, sizeof(float) * p->nparam, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemsetAsync(p->m, 0, sizeof(float) * p->nparam, ctx->stream));
  CK(cudaMemsetAsync(p->v, 0, sizeof(float) * p->nparam, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  p->step = 0;
  return 0;
}

int atlasgpu_mlp_forward(atlasgpu_ctx* ctx, atlasgpu_mlp* p, const float* x, int n, float* y) {
  if (!ctx || !p || !x || !y || n < 1) return fail(ctx, ATLASGPU_EINVAL, "mlp_forward");
  cudaSetDevice(ctx->device);
  int r;
  if ((r = ensure_cap(ctx, p, n))) return r;
  CK(cudaMemcpyAsync(p->x, x, sizeof(float) * (size_t)n * p->nin, cudaMemcpyHostToDevice, ctx->stream));
  if ((r = forward(ctx, p, n))) return r;
  CK(cudaMemcpyAsync(y, p->y, sizeof(float) * (size_t)n * p->nout, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return 0;
}

int atlasgpu_mlp_loss_grad(atlasgpu_ctx* ctx, atlasgpu_mlp* p, const float* x, const float* t, int n,
                           float* grad, float* loss) {
  if (!ctx || !p || !x || !t || n < 1) return fail(ctx, ATLASGPU_EINVAL, "mlp_loss_grad");
  cudaSetDevice(ctx->device);
  int r;
  if ((r = ensure_cap(ctx, p, n))) return r;
  CK(cudaMemcpyAsync(p->x, x, sizeof(float) * (size_t)n * p->nin, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(p->t, t, sizeof(float) * (size_t)n * p->nout, cudaMemcpyHostToDevice, ctx->stream));
  if ((r = forward(ctx, p, n, p->loss)) || (r = backward(ctx, p, n))) return r;
  if (grad) CK(cudaMemcpyAsync(grad, p->g, sizeof(float) * p->nparam, cudaMemcpyDeviceToHost, ctx->stream));
  float l = 0.f;
  CK(cudaMemcpyAsync(&l, p->loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  if (loss) *loss = l;
  return 0;
}

int atlasgpu_mlp_train(atlasgpu_ctx* ctx, atlasgpu_mlp* p, const float* x, const float* t, int n, int epochs,
                       int batch, float lr, uint64_t seed, float* loss_hist) {
  if (!ctx || !p || !x || !t || n < 1 || epochs < 0 || batch < 1)
    return fail(ctx, ATLASGPU_EINVAL, "mlp_train: bad argument");
  cudaSetDevice(ctx->device);
  cudaStream_t st = ctx->stream;
  if (batch > n) batch = n;
  int r;
  if ((r = ensure_cap(ctx, p, batch))) return r;
  float *dx, *dt, *dloss;
  int* didx;
  CK(cudaMalloc(&dx, sizeof(float) * (size_t)n * p->nin));
  CK(cudaMalloc(&dt, sizeof(float) * (size_t)n * p->nout));
  CK(cudaMalloc(&didx, sizeof(int) * (size_t)n));
  CK(cudaMalloc(&dloss, sizeof(float) * (size_t)(epochs + 1)));
  CK(cudaMemcpyAsync(dx, x, sizeof(float) * (size_t)n * p->nin, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(dt, t, sizeof(float) * (size_t)n * p->nout, cudaMemcpyHostToDevice, st));
  std::vector<int> perm(n);
  uint64_t s = seed;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int ep = 0; ep < epochs && r == 0; ++ep) {
    for (int i = 0; i < n; ++i) perm[i] = i;
    for (int i = n - 1; i > 0; --i) {  // Fisher-Yates with splitmix
      const int j = (int)(splitmix(s) % (uint64_t)(i + 1));
      std::swap(perm[i], perm[j]);
    }
    CK(cudaMemcpyAsync(didx, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
    CK(cudaStreamSynchronize(st));  // perm is rewritten next epoch
    for (int b0 = 0; b0 + batch <= n; b0 += batch) {
      k_gather<<<grid_for(ctx, (int64_t)batch * p->nin, 256, 4), 256, 0, st>>>(batch, p->nin, didx + b0, dx, p->x);
      k_gather<<<grid_for(ctx, (int64_t)batch * p->nout, 256, 4), 256, 0, st>>>(batch, p->nout, didx + b0, dt, p->t);
      CKL(ctx);
      if ((r = forward(ctx, p, batch, dloss + ep)) || (r = backward(ctx, p, batch))) break;
      p->step += 1;
      const float c1 = 1.f - powf(b1, (float)p->step), c2 = 1.f - powf(b2, (float)p->step);
      k_adam<<<grid_for(ctx, p->nparam, 256, 4), 256, 0, st>>>(p->nparam, p->w, p->g, p->m, p->v, lr, b1, b2, eps,
                                                               c1, c2);
      CKL(ctx);
    }
  }
  if (r == 0 && loss_hist && epochs > 0)
    CK(cudaMemcpyAsync(loss_hist, dloss, sizeof(float) * epochs, cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  cudaFree(dx);
  cudaFree(dt);
  cudaFree(didx);
  cudaFree(dloss);
  return r;
}

}  // extern "C"
