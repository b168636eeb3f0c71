// Skinny pairs on the SIMT cores (sm_103a): a large operand X (R rows over
// its free modes, K <= 16 contracted) against a small operand W (K x N, N <=
// 16), C[r, n] = sum_k X[r, k] W[k, n].  This is a gate of up to four qubits
// applied to a state vector or a boundary tensor absorbing a gate column:
// memory-bound work whose bytes are X read once and C written once.
//
// One thread per row: it decodes the row's offsets in X and C (the modes are
// merged, so a state-vector row has at most a few), loads its K values of X
// (all in flight at once), multiplies them by W from shared memory (a
// broadcast read) and writes its N results.  Consecutive threads take
// consecutive rows, so each load and store of a warp is coalesced whenever the
// row's first mode has unit stride; when X's unit-stride mode is contracted
// (runs of KV values), a thread reads 16 or 32 aligned bytes at a time instead.
// The offsets of k and n are decoded on the host and come with the launch.
//
// What bounds it: a 16 x 16 row needs 1024 FP32 multiply-adds for 256 bytes,
// 28 us of the FP32 pipes per 2^20 rows against 39 us of HBM, and the broadcast
// reads of W 27 us; with one instruction per multiply-add the issue slots were
// what ran out.  Complex64 rows therefore multiply two columns at a time
// (fma.rn.f32x2).  2^24 amplitudes, 4 qubits: 106 -> 64 us with the unit-stride
// mode contracted, 65 -> 53 otherwise; 3 qubits 72 - 84 -> 48, 2 qubits 54 -> 46.
//
// Accumulation: FP32 for complex64 results (K <= 16 terms; the real part as
// the difference of two sums), FP64 for complex128 results.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "pq_types.cuh"

namespace pq {

namespace {

constexpr int kSkThreads = 128;

struct SkinnyDesc {
  int64_t R;
  int K, N, nr, w64;        // w64: W is complex128
  int64_t rdim[kMaxModes], rsx[kMaxModes], rsc[kMaxModes];
  int32_t rlog[kMaxModes];  // log2 of rdim, or -1
  int64_t kx[kSkinnyK], cn[kSkinnyN];    // offsets of k in X and of n in C
  int64_t kw[kSkinnyK], nw[kSkinnyN];    // offsets of k and n in W
};

// KV consecutive complex64 values (KV * 8 bytes, aligned to them), or one value.
template <int KV, typename TX>
__device__ __forceinline__ void load_run(const TX* p, TX* v) {
  if constexpr (KV == 4) {
    float* f = reinterpret_cast<float*>(v);
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
        : "l"(p));
  } else if constexpr (KV == 2) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = TX{q.x, q.y};
    v[1] = TX{q.z, q.w};
  } else {
    v[0] = __ldg(p);
  }
}

// Offsets of row r in X and C.
__device__ __forceinline__ void row_offsets(const SkinnyDesc& d, int64_t x, int64_t& xo, int64_t& co) {
  xo = co = 0;
  for (int i = 0; i < d.nr; ++i) {
    int64_t q, rem;
    if (d.rlog[i] >= 0) {
      rem = x & (d.rdim[i] - 1);
      q = x >> d.rlog[i];
    } else {
      q = x / d.rdim[i];
      rem = x - q * d.rdim[i];
    }
    xo += rem * d.rsx[i];
    co += rem * d.rsc[i];
    x = q;
  }
}

template <typename R>
__device__ __forceinline__ typename Acc<R>::C w_value(const SkinnyDesc& d, const void* W, int k, int n) {
  if (k >= d.K || n >= d.N) return czero(R());
  const int64_t o = d.kw[k] + d.nw[n];
  return d.w64 ? cvt<R>(static_cast<const double2*>(W)[o]) : cvt<R>(static_cast<const float2*>(W)[o]);
}

// Complex64 X and C.
template <int KMAX, int KV>
__global__ void __launch_bounds__(kSkThreads)
    k_skinny_f(const float2* __restrict__ X, const void* __restrict__ W, float2* __restrict__ C,
               const __grid_constant__ SkinnyDesc d) {
  // columns n, n + 1 of W[k] as (re, re', im, im'), zero past K and N
  __shared__ __align__(16) float w[KMAX][kSkinnyN / 2][4];
  for (int t = threadIdx.x; t < KMAX * kSkinnyN; t += kSkThreads) {
    const int k = t / kSkinnyN, n = t % kSkinnyN;
    const float2 v = w_value<float>(d, W, k, n);
    w[k][n / 2][n & 1] = v.x;
    w[k][n / 2][2 + (n & 1)] = v.y;
  }
  __syncthreads();
  const int64_t step = (int64_t)gridDim.x * kSkThreads;
  for (int64_t r = (int64_t)blockIdx.x * kSkThreads + threadIdx.x; r < d.R; r += step) {
    int64_t xo, co;
    row_offsets(d, r, xo, co);
    float2 a[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; k += KV) {
      if (k < d.K) {
        load_run<KV>(X + xo + d.kx[k], &a[k]);
      } else {
#pragma unroll
        for (int u = 0; u < KV; ++u) a[k + u] = make_float2(0.f, 0.f);
      }
    }
    F2 ax[KMAX], ay[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      ax[k] = f2_dup(a[k].x);
      ay[k] = f2_dup(a[k].y);
    }
    // not unrolled: W is read per group of four columns instead of being kept
    // in registers
#pragma unroll 1
    for (int n0 = 0; n0 < d.N; n0 += 4) {
      F2 rr[2], ii[2], ri[2];  // sums of re re, im im and re im + im re for two column pairs
#pragma unroll
      for (int q = 0; q < 2; ++q) rr[q] = ii[q] = ri[q] = 0;
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(w[k][n0 / 2 + q]);
          rr[q] = f2_fma(ax[k], b.x, rr[q]);
          ii[q] = f2_fma(ay[k], b.y, ii[q]);
          ri[q] = f2_fma(ax[k], b.y, ri[q]);
          ri[q] = f2_fma(ay[k], b.x, ri[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float2 p = f2_get(rr[q]), m = f2_get(ii[q]), y = f2_get(ri[q]);
        if (n0 + 2 * q < d.N) C[co + d.cn[n0 + 2 * q]] = make_float2(p.x - m.x, y.x);
        if (n0 + 2 * q + 1 < d.N) C[co + d.cn[n0 + 2 * q + 1]] = make_float2(p.y - m.y, y.y);
      }
    }
  }
}

// Every other mix of element types (complex128 results in FP64).
template <typename TX, typename TC, int KMAX>
__global__ void __launch_bounds__(kSkThreads)
    k_skinny(const TX* __restrict__ X, const void* __restrict__ W, TC* __restrict__ C,
             const __grid_constant__ SkinnyDesc d) {
  using R = typename std::conditional<std::is_same<TC, double2>::value, double, float>::type;
  using R2 = typename Acc<R>::C;
  __shared__ __align__(16) R2 w[KMAX][kSkinnyN];  // W[k][n], zero past K and N
  for (int t = threadIdx.x; t < KMAX * kSkinnyN; t += kSkThreads)
    w[t / kSkinnyN][t % kSkinnyN] = w_value<R>(d, W, t / kSkinnyN, t % kSkinnyN);
  __syncthreads();
  const int64_t step = (int64_t)gridDim.x * kSkThreads;
  for (int64_t r = (int64_t)blockIdx.x * kSkThreads + threadIdx.x; r < d.R; r += step) {
    int64_t xo, co;
    row_offsets(d, r, xo, co);
    R2 a[KMAX];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) a[k] = k < d.K ? cvt<R>(__ldg(X + xo + d.kx[k])) : czero(R());
#pragma unroll 1
    for (int n0 = 0; n0 < d.N; n0 += 4) {
      R2 acc[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) acc[n] = czero(R());
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
#pragma unroll
        for (int n = 0; n < 4; ++n) cfma(acc[n], a[k], w[k][n0 + n]);
      }
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (n0 + n < d.N) C[co + d.cn[n0 + n]] = store_as<TC>(acc[n]);
    }
  }
}

// Persistent-style grids of the blocks that fit an SM at the kernels' register
// counts (complex64: 64 registers at K <= 16, 46 or fewer below; FP64: 96).
int sk_grid(int64_t rows, int per_sm) {
  return (int)std::min<int64_t>((rows + kSkThreads - 1) / kSkThreads, 152 * per_sm);
}

template <typename TX, typename TC>
cudaError_t launch_mixed(const void* X, const void* W, void* C, const SkinnyDesc& d, cudaStream_t s) {
  if (d.K <= 4)
    k_skinny<TX, TC, 4><<<sk_grid(d.R, 10), kSkThreads, 0, s>>>((const TX*)X, W, (TC*)C, d);
  else
    k_skinny<TX, TC, 16><<<sk_grid(d.R, 5), kSkThreads, 0, s>>>((const TX*)X, W, (TC*)C, d);
  return cudaGetLastError();
}

template <int KMAX>
cudaError_t launch_f(int kv, const void* X, const void* W, void* C, const SkinnyDesc& d, cudaStream_t s) {
  const int grid = sk_grid(d.R, KMAX == 16 ? 8 : 10);
  const float2* x = (const float2*)X;
  if (kv == 4)
    k_skinny_f<KMAX, 4><<<grid, kSkThreads, 0, s>>>(x, W, (float2*)C, d);
  else if (kv == 2)
    k_skinny_f<KMAX, 2><<<grid, kSkThreads, 0, s>>>(x, W, (float2*)C, d);
  else
    k_skinny_f<KMAX, 1><<<grid, kSkThreads, 0, s>>>(x, W, (float2*)C, d);
  return cudaGetLastError();
}

int log2_exact(int64_t v) {
  int l = 0;
  while ((int64_t(1) << l) < v) ++l;
  return (int64_t(1) << l) == v ? l : -1;
}

// Offset of x over n mixed-radix modes.
int64_t offset_of(int64_t x, int n, const int64_t* dim, const int64_t* s) {
  int64_t o = 0;
  for (int i = 0; i < n; ++i) {
    o += x % dim[i] * s[i];
    x /= dim[i];
  }
  return o;
}

}  // namespace

bool skinny_eligible(const GemmDesc& g) {
  return g.Z == 1 && std::max(g.M, g.N) >= kSkinnyMinRows && std::min(g.M, g.N) <= kSkinnyN && g.K <= kSkinnyK;
}

cudaError_t launch_skinny(int ta, int tb, int tc, const void* A, const void* B, void* C, const GemmDesc& g,
                          cudaStream_t stream) {
  if (!skinny_eligible(g)) return cudaErrorInvalidValue;
  // the large side is X (rows), the small side W
  const bool a_big = g.M >= g.N;
  const void* X = a_big ? A : B;
  const void* W = a_big ? B : A;
  const bool x64 = (a_big ? ta : tb) == PQ_C128, c64 = tc == PQ_C128;
  SkinnyDesc d;
  std::memset(&d, 0, sizeof(d));
  d.R = a_big ? g.M : g.N;
  d.N = (int)(a_big ? g.N : g.M);
  d.K = (int)g.K;
  d.w64 = (a_big ? tb : ta) == PQ_C128;
  if (d.R == 0) return cudaSuccess;
  d.nr = a_big ? g.nm : g.nn;
  const int64_t* ksx = a_big ? g.ksa : g.ksb;
  // runs of KV contracted values that are KV * 8 aligned bytes in X: the first
  // K mode has stride 1 and its extent, every other stride and the base are
  // multiples of KV
  int kv = g.nk > 0 && ksx[0] == 1 && !x64 ? 4 : 1;
  auto limit = [&](int64_t v) {
    while (kv > 1 && v % kv) kv /= 2;
  };
  if (kv > 1) {
    limit(g.kdim[0]);
    while (kv > 1 && (uintptr_t)X % (8 * kv)) kv /= 2;
  }
  for (int i = 1; i < g.nk; ++i) limit(ksx[i]);
  for (int i = 0; i < d.nr; ++i) {
    d.rdim[i] = a_big ? g.mdim[i] : g.ndim[i];
    d.rsx[i] = a_big ? g.msa[i] : g.nsb[i];
    d.rsc[i] = a_big ? g.msc[i] : g.nsc[i];
    d.rlog[i] = log2_exact(d.rdim[i]);
    limit(d.rsx[i]);
  }
  for (int k = 0; k < d.K; ++k) {
    d.kx[k] = offset_of(k, g.nk, g.kdim, ksx);
    d.kw[k] = offset_of(k, g.nk, g.kdim, a_big ? g.ksb : g.ksa);
  }
  for (int n = 0; n < d.N; ++n) {
    d.nw[n] = offset_of(n, a_big ? g.nn : g.nm, a_big ? g.ndim : g.mdim, a_big ? g.nsb : g.msa);
    d.cn[n] = offset_of(n, a_big ? g.nn : g.nm, a_big ? g.ndim : g.mdim, a_big ? g.nsc : g.msc);
  }
  if (c64) return x64 ? launch_mixed<double2, double2>(X, W, C, d, stream) : launch_mixed<float2, double2>(X, W, C, d, stream);
  if (x64) return launch_mixed<double2, float2>(X, W, C, d, stream);
  if (d.K <= 4) return launch_f<4>(kv, X, W, C, d, stream);
  if (d.K <= 8) return launch_f<8>(kv, X, W, C, d, stream);
  return launch_f<16>(kv, X, W, C, d, stream);
}

}  // namespace pq
