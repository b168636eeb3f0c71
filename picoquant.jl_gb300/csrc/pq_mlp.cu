// Learned cost model: a small MLP (n_in -> H -> H -> H -> 1, ReLU) trained on
// the GPU with hand-written forward, backward and Adam kernels (FP32 weights),
// with a bf16 inference path.  It predicts log(kernel time) of one pairwise
// contraction from shape features; the planner sums predictions over a plan's
// steps to rank candidate plans.
//
// Layout: activations are row-major [batch x features]; layer l has weights
// W_l [in x out] (row-major) and bias b_l [out].  Parameters are stored in one
// flat FP32 buffer in the order W1 b1 W2 b2 ... so they can be read/written
// as a single array.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "pq_internal.h"

namespace pq {
int check_status(Ctx* ctx);
}
using namespace pq;

namespace {

constexpr int TB = 16;  // tile of the bf16 inference layers

// FP32 layer products on 32 x 32 tiles, 256 threads, four results each, K in
// steps of 128 through shared memory (all of a step's loads in flight at once: 10
// -> 7 us per layer against steps of 32).  A training batch (1024 rows, 128 wide) is
// latency-bound, so the tile is the largest that still gives a block to most
// SMs (128 blocks), and the weight gradients, whose K is the batch, are split
// into chunks of rows (`part`) that k_reduce_parts adds up in order: with K
// walked by 64 blocks they took 61 us per layer, and the bias sums, one thread
// per column over all rows, as long.  Forward and backward of a batch: 19
// launches, 520 us -> 8 launches, 51 us.
constexpr int GT = 32, GTP = GT + 1, GK = 128;

struct Tile32 {
  float a[GK][GTP];  // a[k][m]
  float b[GK][GTP];  // b[k][n]
};
// acc += a^T b over the staged K steps, for rows ty, ty + 16 and columns tx, tx + 16.
__device__ __forceinline__ void tile_fma(const Tile32& t, int kn, int tx, int ty, float (&acc)[2][2]) {
#pragma unroll 8
  for (int k = 0; k < kn; ++k) {
    const float a0 = t.a[k][ty], a1 = t.a[k][ty + 16], b0 = t.b[k][tx], b1 = t.b[k][tx + 16];
    acc[0][0] = fmaf(a0, b0, acc[0][0]);
    acc[0][1] = fmaf(a0, b1, acc[0][1]);
    acc[1][0] = fmaf(a1, b0, acc[1][0]);
    acc[1][1] = fmaf(a1, b1, acc[1][1]);
  }
}

// BACK = false: Y [n x N] = relu(X [n x K] W [K x N] + bias).
// BACK = true:  Y [n x N] = (X [n x K] W^T, W [N x K]), zero where H [n x N] <= 0
// (the gradient through the ReLU of activations H).
template <bool BACK>
__global__ void __launch_bounds__(256)
    k_layer(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
            const float* __restrict__ H, float* __restrict__ Y, int n, int N, int K) {
  __shared__ Tile32 t;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  const int m0 = blockIdx.x * GT, n0 = blockIdx.y * GT;
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (int k0 = 0; k0 < K; k0 += GK) {
    // element e of a step: X and W^T rows along K, W rows along N
    float ra[GT * GK / 256], rb[GT * GK / 256];
#pragma unroll
    for (int i = 0; i < GT * GK / 256; ++i) {
      const int k = lx + 32 * (i & 3), r = ly + 8 * (i >> 2);  // 4 runs of 32 k, rows 8 apart
      ra[i] = m0 + r < n && k0 + k < K ? X[(size_t)(m0 + r) * K + k0 + k] : 0.f;
      if (BACK)
        rb[i] = n0 + r < N && k0 + k < K ? W[(size_t)(n0 + r) * K + k0 + k] : 0.f;
      else
        rb[i] = n0 + lx < N && k0 + ly + 8 * i < K ? W[(size_t)(k0 + ly + 8 * i) * N + n0 + lx] : 0.f;
    }
    if (k0) __syncthreads();  // the previous step has been read
#pragma unroll
    for (int i = 0; i < GT * GK / 256; ++i) {
      const int k = lx + 32 * (i & 3), r = ly + 8 * (i >> 2);
      t.a[k][r] = ra[i];
      if (BACK)
        t.b[k][r] = rb[i];
      else
        t.b[ly + 8 * i][lx] = rb[i];
    }
    __syncthreads();
    tile_fma(t, min(GK, K - k0), tx, ty, acc);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int row = m0 + ty + 16 * i, col = n0 + tx + 16 * j;
      if (row >= n || col >= N) continue;
      const size_t o = (size_t)row * N + col;
      if (BACK)
        Y[o] = H[o] <= 0.f ? 0.f : acc[i][j];
      else {
        const float v = acc[i][j] + bias[col];
        Y[o] = v > 0.f ? v : 0.f;
      }
    }
}

// The output layer (one value per row, a warp each): y = h . w + b.  With
// targets, also the gradient of the mean squared error, dy = 2 (y - t) / n, its
// product with w through the ReLU of h, and the block's sum of squared errors.
__global__ void __launch_bounds__(256)
    k_head(const float* __restrict__ H, const float* __restrict__ w, const float* __restrict__ b, int n, int K,
           float* __restrict__ y, const float* __restrict__ t, float* __restrict__ dy, float* __restrict__ dh,
           float* __restrict__ loss_part) {
  __shared__ float sq[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + warp;
  float e = 0.f;
  if (row < n) {
    const float* h = H + (size_t)row * K;
    float acc = 0.f;
    for (int k = lane; k < K; k += 32) acc = fmaf(h[k], w[k], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    acc += b[0];
    if (lane == 0) y[row] = acc;
    if (t) {
      e = acc - t[row];
      const float g = 2.f * e / (float)n;
      if (lane == 0) dy[row] = g;
      if (dh)
        for (int k = lane; k < K; k += 32) dh[(size_t)row * K + k] = h[k] <= 0.f ? 0.f : g * w[k];
    }
  }
  if (!t) return;
  if (lane == 0) sq[warp] = e * e;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int i = 0; i < 8; ++i) s += sq[i];
    loss_part[blockIdx.x] = s;
  }
}

// Weight and bias gradients of up to kDwLayers layers in one launch:
// part[c][woff ..] = X^T dY and part[c][boff ..] = column sums of dY over chunk c
// of `rows` rows (blockIdx.y), tiles of all layers along blockIdx.x.
constexpr int kDwLayers = 8;
struct DwTable {
  int layers;
  int first[kDwLayers + 1];  // tiles before each layer
  int M[kDwLayers], N[kDwLayers];
  int64_t woff[kDwLayers], boff[kDwLayers];
  const float* x[kDwLayers];
  const float* dy[kDwLayers];
};
__global__ void __launch_bounds__(256)
    k_dw(const __grid_constant__ DwTable d, int n, int rows, int64_t n_params, float* __restrict__ part) {
  __shared__ Tile32 t;
  int l = 0;
  while (l + 1 < d.layers && d.first[l + 1] <= (int)blockIdx.x) ++l;
  const int M = d.M[l], N = d.N[l], nt = (N + GT - 1) / GT, id = (int)blockIdx.x - d.first[l];
  const int m0 = id / nt * GT, n0 = id % nt * GT;
  const float *X = d.x[l], *D = d.dy[l];
  const int r0 = blockIdx.y * rows, r1 = min(n, r0 + rows);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int lx = threadIdx.x & 31, ly = threadIdx.x >> 5;
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  float col = 0.f;  // threads 0 .. 31 of the first row of tiles: a column's sum
  for (int k0 = r0; k0 < r1; k0 += GK) {
    float ra[GT * GK / 256], rb[GT * GK / 256];
#pragma unroll
    for (int i = 0; i < GT * GK / 256; ++i) {
      const int r = ly + 8 * i;
      const bool in = k0 + r < r1;
      ra[i] = in && m0 + lx < M ? X[(size_t)(k0 + r) * M + m0 + lx] : 0.f;
      rb[i] = in && n0 + lx < N ? D[(size_t)(k0 + r) * N + n0 + lx] : 0.f;
    }
    if (k0 != r0) __syncthreads();  // the previous step has been read
#pragma unroll
    for (int i = 0; i < GT * GK / 256; ++i) {
      t.a[ly + 8 * i][lx] = ra[i];
      t.b[ly + 8 * i][lx] = rb[i];
    }
    __syncthreads();
    const int kn = min(GK, r1 - k0);
    tile_fma(t, kn, tx, ty, acc);
    if (m0 == 0 && threadIdx.x < GT)
      for (int k = 0; k < kn; ++k) col += t.b[k][threadIdx.x];
  }
  float* P = part + blockIdx.y * n_params;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = m0 + ty + 16 * i, c = n0 + tx + 16 * j;
      if (r < M && c < N) P[d.woff[l] + (int64_t)r * N + c] = acc[i][j];
    }
  if (m0 == 0 && threadIdx.x < GT && n0 + (int)threadIdx.x < N) P[d.boff[l] + n0 + threadIdx.x] = col;
}

// g[i] = sum of the chunks' parts in order; the last block adds up the loss.
__global__ void __launch_bounds__(256)
    k_reduce_parts(const float* __restrict__ part, int chunks, int64_t n_params, float* __restrict__ g,
                   const float* __restrict__ loss_part, int n_loss, int n, float* __restrict__ loss) {
  if (blockIdx.x + 1 < gridDim.x) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_params) return;
    float s = 0.f;
    for (int c = 0; c < chunks; ++c) s += part[c * n_params + i];
    g[i] = s;
    return;
  }
  __shared__ float sm[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < n_loss; i += 256) s += loss_part[i];
  sm[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sm[threadIdx.x] += sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = sm[0] / (float)n;
}

// Inference layer in bf16: weights and inputs rounded to bf16, FP32 accumulate.
__global__ void k_bf16_layer(const __nv_bfloat16* __restrict__ X, const __nv_bfloat16* __restrict__ W,
                             const float* __restrict__ bias, __nv_bfloat16* __restrict__ Y, float* __restrict__ yf,
                             int M, int N, int K, int relu) {
  __shared__ float Xs[TB][TB + 1];
  __shared__ float Ws[TB][TB + 1];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int row = blockIdx.y * TB + ty, col = blockIdx.x * TB + tx;
  float acc = 0.f;
  for (int k0 = 0; k0 < K; k0 += TB) {
    int ka = k0 + tx, kb = k0 + ty;
    Xs[ty][tx] = (row < M && ka < K) ? __bfloat162float(X[(size_t)row * K + ka]) : 0.f;
    Ws[ty][tx] = (col < N && kb < K) ? __bfloat162float(W[(size_t)kb * N + col]) : 0.f;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TB; ++k) acc = fmaf(Xs[ty][k], Ws[k][tx], acc);
    __syncthreads();
  }
  if (row < M && col < N) {
    acc += bias[col];
    if (relu) acc = acc > 0.f ? acc : 0.f;
    if (Y) Y[(size_t)row * N + col] = __float2bfloat16(acc);
    if (yf) yf[(size_t)row * N + col] = acc;
  }
}

// Gather training rows by index into the batch buffers.
__global__ void k_gather_rows(const float* __restrict__ X, const float* __restrict__ Y,
                              const int64_t* __restrict__ idx, int b, int n_in, float* __restrict__ xb,
                              float* __restrict__ yb) {
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= b) return;
  int64_t src = idx[r];
  for (int j = 0; j < n_in; ++j) xb[(size_t)r * n_in + j] = X[(size_t)src * n_in + j];
  yb[r] = Y[src];
}

__global__ void k_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int64_t n, float lr, float b1, float b2, float eps, float c1, float c2) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gi = g[i];
  float mi = b1 * m[i] + (1.f - b1) * gi;
  float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}


// Gradients of up to this many bytes are read back through a pinned buffer of
// the handle: a copy into the caller's pageable memory is staged and waited
// for inside the driver (136 KB of gradients, batch of 1024: 92 -> 88 us).  Larger
// ones, where the copy itself is the time, go straight to the caller.
constexpr size_t kPinnedGrad = 1 << 20;

}  // namespace

struct pq_mlp {
  Ctx* ctx = nullptr;
  int n_in = 0, hidden = 0, layers = 0;  // `layers` hidden layers + 1 output layer
  std::vector<int> din, dout;            // per linear layer
  std::vector<int64_t> woff, boff;       // offsets in the flat parameter buffer
  int64_t n_params = 0;
  float* d_p = nullptr;
  float* d_g = nullptr;  // gradients, then the loss (read together)
  float* h_g = nullptr;  // pinned host copy of d_g (small models)
  float* d_m = nullptr;
  float* d_v = nullptr;
  int64_t step = 0;
  // workspace for a batch
  int cap = 0;       // rows that the activations hold
  int grad_cap = 0;  // rows that the gradient workspace holds
  std::vector<float*> act;  // act[0] = input, act[l+1] = output of layer l
  std::vector<float*> dact;
  float* d_t = nullptr;
  float* d_loss = nullptr;
  float* d_part = nullptr;       // weight-gradient chunks (at most max_chunks x n_params)
  float* d_loss_part = nullptr;  // squared errors per k_head block
  __nv_bfloat16* d_wbf = nullptr;
  __nv_bfloat16* d_xb[2] = {nullptr, nullptr};
};

namespace {

// The batch in chunks of rows for the weight gradients: 128 rows each, at most
// 64 chunks and kPartBytes of partial gradients (a model whose gradients are
// large has tiles for every SM without chunks).
constexpr int64_t kPartBytes = 64 << 20;
int max_chunks(int64_t n_params) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(64, kPartBytes / (n_params * (int64_t)sizeof(float))));
}
int chunk_rows(int n, int64_t n_params) {
  const int c = max_chunks(n_params);
  return std::max(128, ((n + c - 1) / c + GT - 1) / GT * GT);
}

void free_ws(pq_mlp* m) {
  for (auto p : m->act) cudaFree(p);
  for (auto p : m->dact) cudaFree(p);
  m->act.clear();
  m->dact.clear();
  cudaFree(m->d_t);
  cudaFree(m->d_xb[0]);
  cudaFree(m->d_xb[1]);
  m->d_t = nullptr;
  m->d_xb[0] = m->d_xb[1] = nullptr;
  m->cap = 0;
}
void free_grad_ws(pq_mlp* m) {
  cudaFree(m->d_part);
  cudaFree(m->d_loss_part);
  m->d_part = m->d_loss_part = nullptr;
  m->grad_cap = 0;
}

int ensure_ws(pq_mlp* m, int n) {
  if (n <= m->cap) return PQ_OK;
  free_ws(m);
  const int L = (int)m->din.size();
  m->act.assign(L + 1, nullptr);
  m->dact.assign(L + 1, nullptr);
  cudaError_t e = cudaSuccess;
  for (int l = 0; l <= L; ++l) {
    int w = l == 0 ? m->n_in : m->dout[l - 1];
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->act[l], sizeof(float) * (size_t)n * w);
    if (e == cudaSuccess) e = cudaMalloc((void**)&m->dact[l], sizeof(float) * (size_t)n * w);
  }
  int wmax = std::max(m->n_in, m->hidden);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_t, sizeof(float) * (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_xb[0], sizeof(__nv_bfloat16) * (size_t)n * wmax);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_xb[1], sizeof(__nv_bfloat16) * (size_t)n * wmax);
  if (e != cudaSuccess) {
    free_ws(m);
    return cuda_fail(m->ctx, e, "mlp workspace");
  }
  m->cap = n;
  return PQ_OK;
}
// What gradients of n rows need beside the activations (inference does not).
int ensure_grad_ws(pq_mlp* m, int n) {
  if (n <= m->grad_cap) return PQ_OK;
  free_grad_ws(m);
  // (a smaller batch has no more chunks than this)
  const size_t chunks = (size_t)std::min(max_chunks(m->n_params), (n + 127) / 128);
  cudaError_t e = cudaMalloc((void**)&m->d_part, sizeof(float) * (size_t)m->n_params * chunks);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_loss_part, sizeof(float) * (size_t)((n + 7) / 8));
  if (e != cudaSuccess) {
    free_grad_ws(m);
    return cuda_fail(m->ctx, e, "mlp gradient workspace");
  }
  m->grad_cap = n;
  return PQ_OK;
}

// Forward pass (FP32) over n rows already in act[0]; with targets (d_t), the
// output layer's kernel also starts the backward pass.
void forward(pq_mlp* m, int n, bool train) {
  const int L = (int)m->din.size();
  cudaStream_t s = m->ctx->stream;
  for (int l = 0; l + 1 < L; ++l) {
    dim3 grid((n + GT - 1) / GT, (m->dout[l] + GT - 1) / GT);
    k_layer<false><<<grid, 256, 0, s>>>(m->act[l], m->d_p + m->woff[l], m->d_p + m->boff[l], nullptr, m->act[l + 1], n,
                                        m->dout[l], m->din[l]);
  }
  k_head<<<(n + 7) / 8, 256, 0, s>>>(m->act[L - 1], m->d_p + m->woff[L - 1], m->d_p + m->boff[L - 1], n, m->din[L - 1],
                                     m->act[L], train ? m->d_t : nullptr, m->dact[L], L > 1 ? m->dact[L - 1] : nullptr,
                                     m->d_loss_part);
}

// Backward pass after forward(train): gradients of the mean squared error into
// d_g; returns with the loss in d_loss (device).
void backward(pq_mlp* m, int n) {
  const int L = (int)m->din.size();
  cudaStream_t s = m->ctx->stream;
  // dact[l] = dact[l+1] W_l^T, masked by ReLU of act[l] (k_head wrote dact[L-1])
  for (int l = L - 2; l > 0; --l) {
    dim3 grid((n + GT - 1) / GT, (m->din[l] + GT - 1) / GT);
    k_layer<true><<<grid, 256, 0, s>>>(m->dact[l + 1], m->d_p + m->woff[l], nullptr, m->act[l], m->dact[l], n,
                                       m->din[l], m->dout[l]);
  }
  const int rows = chunk_rows(n, m->n_params), chunks = (n + rows - 1) / rows;
  for (int l0 = 0; l0 < L; l0 += kDwLayers) {
    DwTable d;
    d.layers = std::min(kDwLayers, L - l0);
    d.first[0] = 0;
    for (int i = 0; i < d.layers; ++i) {
      const int l = l0 + i;
      d.M[i] = m->din[l];
      d.N[i] = m->dout[l];
      d.woff[i] = m->woff[l];
      d.boff[i] = m->boff[l];
      d.x[i] = m->act[l];
      d.dy[i] = m->dact[l + 1];
      d.first[i + 1] = d.first[i] + ((d.M[i] + GT - 1) / GT) * ((d.N[i] + GT - 1) / GT);
    }
    k_dw<<<dim3(d.first[d.layers], chunks), 256, 0, s>>>(d, n, rows, m->n_params, m->d_part);
  }
  k_reduce_parts<<<(unsigned)((m->n_params + 255) / 256) + 1, 256, 0, s>>>(m->d_part, chunks, m->n_params, m->d_g,
                                                                         m->d_loss_part, (n + 7) / 8, n, m->d_loss);
}

}  // namespace

extern "C" {

int pq_mlp_create(pq_ctx* c, int n_in, int hidden, int hidden_layers, uint64_t seed, pq_mlp** out) {
  if (!c || !out || n_in < 1 || hidden < 1 || hidden_layers < 1) return PQ_ERR_INVALID;
  Ctx* ctx = &c->impl;
  pq_mlp* m = new pq_mlp();
  m->ctx = ctx;
  m->n_in = n_in;
  m->hidden = hidden;
  m->layers = hidden_layers;
  int w = n_in;
  for (int l = 0; l < hidden_layers; ++l) {
    m->din.push_back(w);
    m->dout.push_back(hidden);
    w = hidden;
  }
  m->din.push_back(w);
  m->dout.push_back(1);
  for (size_t l = 0; l < m->din.size(); ++l) {
    m->woff.push_back(m->n_params);
    m->n_params += (int64_t)m->din[l] * m->dout[l];
    m->boff.push_back(m->n_params);
    m->n_params += m->dout[l];
  }
  // He-uniform initialisation (host, seeded), zero biases
  std::vector<float> h((size_t)m->n_params, 0.f);
  std::mt19937_64 rng(seed);
  for (size_t l = 0; l < m->din.size(); ++l) {
    float a = std::sqrt(6.f / (float)m->din[l]);
    std::uniform_real_distribution<float> U(-a, a);
    for (int64_t i = 0; i < (int64_t)m->din[l] * m->dout[l]; ++i) h[m->woff[l] + i] = U(rng);
  }
  cudaError_t e = cudaMalloc((void**)&m->d_p, sizeof(float) * m->n_params);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_g, sizeof(float) * (m->n_params + 1));
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_m, sizeof(float) * m->n_params);
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_v, sizeof(float) * m->n_params);
  if (e == cudaSuccess) m->d_loss = m->d_g + m->n_params;
  if (e == cudaSuccess) e = cudaMalloc((void**)&m->d_wbf, sizeof(__nv_bfloat16) * m->n_params);
  const size_t gbytes = sizeof(float) * ((size_t)m->n_params + 1);
  if (e == cudaSuccess && gbytes <= kPinnedGrad) e = cudaHostAlloc((void**)&m->h_g, gbytes, cudaHostAllocDefault);
  if (e == cudaSuccess) e = cudaMemcpy(m->d_p, h.data(), sizeof(float) * m->n_params, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(m->d_m, 0, sizeof(float) * m->n_params);
  if (e == cudaSuccess) e = cudaMemset(m->d_v, 0, sizeof(float) * m->n_params);
  if (e != cudaSuccess) {
    cudaFree(m->d_p);
    cudaFree(m->d_g);
    cudaFree(m->d_m);
    cudaFree(m->d_v);
    cudaFree(m->d_wbf);
    if (m->h_g) cudaFreeHost(m->h_g);
    delete m;
    return cuda_fail(ctx, e, "mlp create");
  }
  *out = m;
  return PQ_OK;
}

int pq_mlp_destroy(pq_mlp* m) {
  if (!m) return PQ_ERR_INVALID;
  cudaStreamSynchronize(m->ctx->stream);
  free_ws(m);
  free_grad_ws(m);
  cudaFree(m->d_p);
  cudaFree(m->d_g);
  cudaFree(m->d_m);
  cudaFree(m->d_v);
  cudaFree(m->d_wbf);
  if (m->h_g) cudaFreeHost(m->h_g);
  delete m;
  return PQ_OK;
}

int pq_mlp_num_params(pq_mlp* m, int64_t* n) {
  if (!m || !n) return PQ_ERR_INVALID;
  *n = m->n_params;
  return PQ_OK;
}

int pq_mlp_get_params(pq_mlp* m, float* w, int64_t n) {
  if (!m || !w || n < m->n_params) return PQ_ERR_INVALID;
  cudaError_t e = cudaMemcpyAsync(w, m->d_p, sizeof(float) * m->n_params, cudaMemcpyDeviceToHost, m->ctx->stream);
  if (e != cudaSuccess) return cuda_fail(m->ctx, e, "mlp get params");
  return check_status(m->ctx);
}

int pq_mlp_set_params(pq_mlp* m, const float* w, int64_t n) {
  if (!m || !w || n != m->n_params) return PQ_ERR_INVALID;
  cudaError_t e = cudaMemcpyAsync(m->d_p, w, sizeof(float) * m->n_params, cudaMemcpyHostToDevice, m->ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->d_m, 0, sizeof(float) * m->n_params, m->ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->d_v, 0, sizeof(float) * m->n_params, m->ctx->stream);
  if (e != cudaSuccess) return cuda_fail(m->ctx, e, "mlp set params");
  m->step = 0;
  return check_status(m->ctx);
}

int pq_mlp_gradients(pq_mlp* m, const float* X, const float* y, int64_t n, float* grad, float* loss) {
  if (!m || !X || !y || !grad || n < 1 || n > (1 << 24)) return PQ_ERR_INVALID;
  int st = ensure_ws(m, (int)n);
  if (!st) st = ensure_grad_ws(m, (int)n);
  if (st) return st;
  cudaStream_t s = m->ctx->stream;
  cudaMemcpyAsync(m->act[0], X, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(m->d_t, y, sizeof(float) * n, cudaMemcpyHostToDevice, s);
  forward(m, (int)n, true);
  backward(m, (int)n);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(m->ctx, e, "mlp gradients");
  // through the handle's pinned buffer where it has one (kPinnedGrad)
  const size_t bytes = sizeof(float) * (size_t)m->n_params;
  float l = 0;
  if (m->h_g) {
    e = cudaMemcpyAsync(m->h_g, m->d_g, bytes + sizeof(float), cudaMemcpyDeviceToHost, s);
  } else {
    e = cudaMemcpyAsync(grad, m->d_g, bytes, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&l, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s);
  }
  if (e != cudaSuccess) return cuda_fail(m->ctx, e, "mlp gradients");
  st = check_status(m->ctx);
  if (st) return st;
  if (m->h_g) {
    std::memcpy(grad, m->h_g, bytes);
    l = m->h_g[m->n_params];
  }
  if (loss) *loss = l;
  return PQ_OK;
}

int pq_mlp_train(pq_mlp* m, const float* X, const float* y, int64_t n, int epochs, int batch, float lr,
                 uint64_t seed, float* final_loss) {
  if (!m || !X || !y || n < 1 || epochs < 1 || batch < 1) return PQ_ERR_INVALID;
  Ctx* ctx = m->ctx;
  cudaStream_t s = ctx->stream;
  // the whole data set lives on the device; batches are gathered by index
  float *dX = nullptr, *dY = nullptr;
  int64_t* dperm = nullptr;
  cudaError_t e = cudaMalloc((void**)&dX, sizeof(float) * n * m->n_in);
  if (e == cudaSuccess) e = cudaMalloc((void**)&dY, sizeof(float) * n);
  if (e == cudaSuccess) e = cudaMalloc((void**)&dperm, sizeof(int64_t) * n);
  if (e != cudaSuccess) {
    cudaFree(dX);
    cudaFree(dY);
    return cuda_fail(ctx, e, "mlp train data");
  }
  cudaMemcpyAsync(dX, X, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(dY, y, sizeof(float) * n, cudaMemcpyHostToDevice, s);
  const int b = (int)std::min<int64_t>(batch, n);
  int st = ensure_ws(m, b);
  if (!st) st = ensure_grad_ws(m, b);
  if (st) {
    cudaFree(dX);
    cudaFree(dY);
    cudaFree(dperm);
    return st;
  }
  std::mt19937_64 rng(seed);
  std::vector<int64_t> perm(n);
  for (int64_t i = 0; i < n; ++i) perm[i] = i;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  float last = 0.f;
  for (int ep = 0; ep < epochs; ++ep) {
    std::shuffle(perm.begin(), perm.end(), rng);
    // contiguous shuffled chunks: copy rows with one memcpy per chunk of the
    // permutation (rows are small, so gather on the host-side index list)
    e = cudaMemcpyAsync(dperm, perm.data(), sizeof(int64_t) * n, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) break;
    for (int64_t i0 = 0; i0 + b <= n; i0 += b) {
      k_gather_rows<<<(b + 127) / 128, 128, 0, s>>>(dX, dY, dperm + i0, b, m->n_in, m->act[0], m->d_t);
      forward(m, b, true);
      backward(m, b);
      ++m->step;
      float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
      k_adam<<<(unsigned)((m->n_params + 255) / 256), 256, 0, s>>>(m->d_p, m->d_g, m->d_m, m->d_v, m->n_params, lr,
                                                                    b1, b2, eps, c1, c2);
    }
    e = cudaMemcpyAsync(&last, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) break;
  }
  cudaFree(dX);
  cudaFree(dY);
  cudaFree(dperm);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "mlp train");
  if (final_loss) *final_loss = last;
  return check_status(ctx);
}

int pq_mlp_predict(pq_mlp* m, const float* X, int64_t n, float* out, int bf16) {
  if (!m || !X || !out || n < 1 || n > (1 << 24)) return PQ_ERR_INVALID;
  int st = ensure_ws(m, (int)n);
  if (st) return st;
  cudaStream_t s = m->ctx->stream;
  const int L = (int)m->din.size();
  cudaMemcpyAsync(m->act[0], X, sizeof(float) * n * m->n_in, cudaMemcpyHostToDevice, s);
  if (!bf16) {
    forward(m, (int)n, false);
  } else {
    k_to_bf16<<<(unsigned)((m->n_params + 255) / 256), 256, 0, s>>>(m->d_p, m->d_wbf, m->n_params);
    k_to_bf16<<<(unsigned)((n * m->n_in + 255) / 256), 256, 0, s>>>(m->act[0], m->d_xb[0], n * m->n_in);
    int cur = 0;
    for (int l = 0; l < L; ++l) {
      dim3 blk(TB, TB), grd((m->dout[l] + TB - 1) / TB, (unsigned)((n + TB - 1) / TB));
      const bool last = l + 1 == L;
      k_bf16_layer<<<grd, blk, 0, s>>>(m->d_xb[cur], m->d_wbf + m->woff[l], m->d_p + m->boff[l],
                                        last ? nullptr : m->d_xb[1 - cur], last ? m->act[L] : nullptr, (int)n,
                                        m->dout[l], m->din[l], last ? 0 : 1);
      cur = 1 - cur;
    }
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(m->ctx, e, "mlp predict");
  return download(m->ctx, out, m->act[L], sizeof(float) * n, "mlp predict");
}

}  // extern "C"
