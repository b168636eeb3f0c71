// Skinny pairs on the SIMT cores (sm_103a): a large operand X (R rows over
// its free modes, K <= 16 contracted) against a small operand W (K x N, N <=
// 128), C[r, n, z] = sum_k X[r, k, z] W[k, n, z].  This is a gate of up to four
// qubits applied to a state vector or a boundary tensor absorbing a gate column
// (with a batch index z, for every bitstring or slice): memory-bound work whose
// bytes are X read once and C written once.
//
// One thread per row: it decodes the row's offsets in X and C (the modes are
// merged, so a state-vector row has at most a few), loads its K values of X
// (all in flight at once), multiplies them by W from shared memory (a
// broadcast read) and writes its N results.  Consecutive threads take
// consecutive rows, so each load and store of a warp is coalesced whenever the
// row's first mode has unit stride; when X's unit-stride mode is contracted
// (runs of KV values), a thread reads 16 or 32 aligned bytes at a time instead.
// The offsets of k and n are decoded on the host and come with the launch.  The
// batch is the grid's y: one z and its W per block.  Where the small operand's
// fastest mode is the result's, four columns are one aligned store.
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
// FP64 rows are bound by the multiply-adds (2 per clock and SM), so what counts
// is that every SM gets the same number of rows: 2^16 rows in blocks of 128 are 3
// or 4 per SM, in blocks of 64 they are 6 or 7 (2^18 amplitudes, 4 qubits: 72 ->
// 41 us, 2^20: 135 -> 128), and that K is not padded (2^20, 3 qubits: 135 -> 62).
constexpr int kSkThreads64 = 64;

struct SkinnyDesc {
  int64_t R, Z;
  int K, N, nr, nz;
  int cols;                 // columns per block (blockIdx.z)
  int w64;                  // W is complex128
  int cvec;                 // columns 4i .. 4i + 3 are 32 aligned bytes of C (complex64)
  int64_t rdim[kMaxModes], rsx[kMaxModes], rsc[kMaxModes];
  int32_t rlog[kMaxModes];  // log2 of rdim, or -1
  int64_t zdim[kMaxModes], zsx[kMaxModes], zsw[kMaxModes], zsc[kMaxModes];
  int64_t kx[kSkinnyK], cn[kSkinnyN];    // offsets of k in X and of n in C
  int64_t kw[kSkinnyK], nw[kSkinnyN];    // offsets of k and n in W
};
static_assert(sizeof(SkinnyDesc) + 64 <= 32764, "kernel parameters");

// Offset of x over n mixed-radix modes.
__host__ __device__ inline int64_t offset_of(int64_t x, int n, const int64_t* dim, const int64_t* s) {
  int64_t o = 0;
  for (int i = 0; i < n; ++i) {
    o += x % dim[i] * s[i];
    x /= dim[i];
  }
  return o;
}

// Offsets of batch index z in X, W and C.
__device__ __forceinline__ void batch_offsets(const SkinnyDesc& d, int64_t z, int64_t& zx, int64_t& zw, int64_t& zc) {
  zx = zw = zc = 0;
  for (int i = 0; i < d.nz; ++i) {
    const int64_t q = z / d.zdim[i], rem = z - q * d.zdim[i];
    zx += rem * d.zsx[i];
    zw += rem * d.zsw[i];
    zc += rem * d.zsc[i];
    z = q;
  }
}

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
__device__ __forceinline__ typename Acc<R>::C w_value(const SkinnyDesc& d, const void* W, int64_t zw, int k, int n) {
  if (k >= d.K || n >= d.N) return czero(R());
  const int64_t o = zw + d.kw[k] + d.nw[n];
  return d.w64 ? cvt<R>(static_cast<const double2*>(W)[o]) : cvt<R>(static_cast<const float2*>(W)[o]);
}

// One row of complex64 X: its K values (zero past K) and its products with W's
// columns n0 .. n0 + 3 (columns n, n + 1 of W[k] as (re, re', im, im') at
// w[(k * np + n / 2) * 4]).
template <int KMAX, int KV>
__device__ __forceinline__ void load_row(const SkinnyDesc& d, const float2* x, F2* ax, F2* ay) {
  float2 a[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; k += KV) {
    if (k < d.K) {
      load_run<KV>(x + d.kx[k], &a[k]);
    } else {
#pragma unroll
      for (int u = 0; u < KV; ++u) a[k + u] = make_float2(0.f, 0.f);
    }
  }
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
    ax[k] = f2_dup(a[k].x);
    ay[k] = f2_dup(a[k].y);
  }
}
// The real part's two sums stay apart and meet in one subtraction (fewer
// instructions, and chains half as long: rms error 9.3e-8 instead of 1.04e-7 for
// K = 16); for K <= 4 they are one chain, where the subtraction's own rounding
// would count (K = 2: 4.5e-8 against 4.2e-8).
template <int KMAX>
__device__ __forceinline__ void four_columns(const F2* ax, const F2* ay, const float* w, int np, int n0, float2* o) {
  F2 rr[2], ii[2], ri[2];  // sums of re re, im im and re im + im re for two column pairs
#pragma unroll
  for (int q = 0; q < 2; ++q) rr[q] = ii[q] = ri[q] = 0;
#pragma unroll
  for (int k = 0; k < KMAX; ++k) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(w + (k * np + n0 / 2 + q) * 4);
      rr[q] = f2_fma(ax[k], b.x, rr[q]);
      if constexpr (KMAX <= 4)
        rr[q] = f2_fma(ay[k] ^ 0x8000000080000000ull, b.y, rr[q]);
      else
        ii[q] = f2_fma(ay[k], b.y, ii[q]);
      ri[q] = f2_fma(ax[k], b.y, ri[q]);
      ri[q] = f2_fma(ay[k], b.x, ri[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float2 p = f2_get(rr[q]), m = f2_get(ii[q]), y = f2_get(ri[q]);
    o[2 * q] = make_float2(p.x - m.x, y.x);
    o[2 * q + 1] = make_float2(p.y - m.y, y.y);
  }
}
__device__ __forceinline__ void w_store(float* w, int np, int k, int n, float2 v) {
  float* e = w + (k * np + n / 2) * 4 + (n & 1);
  e[0] = v.x;
  e[2] = v.y;
}

// Complex64 X and C, up to 16 columns, no batch.
template <int KMAX, int KV>
__global__ void __launch_bounds__(kSkThreads)
    k_skinny_f(const float2* __restrict__ X, const void* __restrict__ W, float2* __restrict__ C,
               const __grid_constant__ SkinnyDesc d) {
  constexpr int NP = 8;
  __shared__ __align__(16) float w[KMAX * NP * 4];  // zero past K and N
  for (int t = threadIdx.x; t < KMAX * 2 * NP; t += kSkThreads)
    w_store(w, NP, t / (2 * NP), t % (2 * NP), w_value<float>(d, W, 0, t / (2 * NP), t % (2 * NP)));
  __syncthreads();
  const int64_t step = (int64_t)gridDim.x * kSkThreads;
  for (int64_t r = (int64_t)blockIdx.x * kSkThreads + threadIdx.x; r < d.R; r += step) {
    int64_t xo, co;
    row_offsets(d, r, xo, co);
    F2 ax[KMAX], ay[KMAX];
    load_row<KMAX, KV>(d, X + xo, ax, ay);
    // not unrolled: W is read per group of four columns instead of being kept
    // in registers
#pragma unroll 1
    for (int n0 = 0; n0 < d.N; n0 += 4) {
      float2 o[4];
      four_columns<KMAX>(ax, ay, w, NP, n0, o);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (n0 + n < d.N) C[co + d.cn[n0 + n]] = o[n];
    }
  }
}

// Complex64 X and C, any number of columns up to 128, batched, or with whole
// columns adjacent in C.
template <int KMAX, int KV>
__global__ void __launch_bounds__(kSkThreads)
    k_skinny_w(const float2* __restrict__ X, const void* __restrict__ W, float2* __restrict__ C,
               const __grid_constant__ SkinnyDesc d) {
  extern __shared__ __align__(16) float w[];  // KMAX * np * 4, zero past K and N
  const int nb = blockIdx.z * d.cols, ne = min(d.N, nb + d.cols);  // this block's columns
  const int np = (ne - nb + 3) / 4 * 2;
  const int64_t step = (int64_t)gridDim.x * kSkThreads;
  for (int64_t z = blockIdx.y; z < d.Z; z += gridDim.y) {
    int64_t zx, zw, zc;
    batch_offsets(d, z, zx, zw, zc);
    if (z != blockIdx.y) __syncthreads();  // the previous W has been read
    for (int t = threadIdx.x; t < KMAX * 2 * np; t += kSkThreads) {
      const int k = t / (2 * np), n = t - k * (2 * np);
      w_store(w, np, k, n, w_value<float>(d, W, zw, k, nb + n));
    }
    __syncthreads();
    for (int64_t r = (int64_t)blockIdx.x * kSkThreads + threadIdx.x; r < d.R; r += step) {
      int64_t xo, co;
      row_offsets(d, r, xo, co);
      F2 ax[KMAX], ay[KMAX];
      load_row<KMAX, KV>(d, X + zx + xo, ax, ay);
      float2* c = C + zc + co;
#pragma unroll 1
      for (int n0 = nb; n0 < ne; n0 += 4) {
        float2 o[4];
        four_columns<KMAX>(ax, ay, w, np, n0 - nb, o);
        if (d.cvec) {
          asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(c + d.cn[n0]), "f"(o[0].x), "f"(o[0].y),
                       "f"(o[1].x), "f"(o[1].y), "f"(o[2].x), "f"(o[2].y), "f"(o[3].x), "f"(o[3].y)
                       : "memory");
        } else {
#pragma unroll
          for (int n = 0; n < 4; ++n)
            if (n0 + n < ne) c[d.cn[n0 + n]] = o[n];
        }
      }
    }
  }
}

// Every other mix of element types (complex128 results in FP64).  ONE: a column
// at a time, else four (padded: 2^18 rows, N = 1, K = 4 in 35 us so, 13 with ONE).
template <typename TX, typename TC, int KMAX, bool ONE>
__global__ void __launch_bounds__(kSkThreads64)
    k_skinny(const TX* __restrict__ X, const void* __restrict__ W, TC* __restrict__ C,
             const __grid_constant__ SkinnyDesc d) {
  using R = typename std::conditional<std::is_same<TC, double2>::value, double, float>::type;
  using R2 = typename Acc<R>::C;
  // W[k][n] of this block's columns at w[k * nw + n], zero past K and N (nw a multiple of four)
  extern __shared__ __align__(16) unsigned char w_raw[];
  R2* w = reinterpret_cast<R2*>(w_raw);
  const int nb = blockIdx.z * d.cols, ne = min(d.N, nb + d.cols);
  const int nw = (ne - nb + 3) / 4 * 4;
  const int64_t step = (int64_t)gridDim.x * kSkThreads64;
  for (int64_t z = blockIdx.y; z < d.Z; z += gridDim.y) {
    int64_t zx, zw, zc;
    batch_offsets(d, z, zx, zw, zc);
    if (z != blockIdx.y) __syncthreads();  // the previous W has been read
    for (int t = threadIdx.x; t < KMAX * nw; t += kSkThreads64) w[t] = w_value<R>(d, W, zw, t / nw, nb + t % nw);
    __syncthreads();
    for (int64_t r = (int64_t)blockIdx.x * kSkThreads64 + threadIdx.x; r < d.R; r += step) {
      int64_t xo, co;
      row_offsets(d, r, xo, co);
      xo += zx;
      co += zc;
      R2 a[KMAX];
#pragma unroll
      for (int k = 0; k < KMAX; ++k) a[k] = k < d.K ? cvt<R>(__ldg(X + xo + d.kx[k])) : czero(R());
      constexpr int CG = ONE ? 1 : 4;
#pragma unroll 1
      for (int n0 = nb; n0 < ne; n0 += CG) {
        R2 acc[CG];
#pragma unroll
        for (int n = 0; n < CG; ++n) acc[n] = czero(R());
#pragma unroll
        for (int k = 0; k < KMAX; ++k) {
          if (k < d.K) {  // (uniform: no FP64 time for padding)
#pragma unroll
            for (int n = 0; n < CG; ++n) cfma(acc[n], a[k], w[k * nw + n0 - nb + n]);
          }
        }
#pragma unroll
        for (int n = 0; n < CG; ++n)
          if (n0 + n < ne) C[co + d.cn[n0 + n]] = store_as<TC>(acc[n]);
      }
    }
  }
}

// Narrow pairs with a longer K (complex64 results): one thread per row again, up
// to 8 columns of W per block (blockIdx.y; with 16 the compensated sums leave
// three blocks per SM: 2^16 rows, N = 16, K = 128 in 82 us against 60), K in
// steps of 128 through shared memory.  Each 16 terms are summed in FP32 and
// folded into a compensated sum per column, as the tiled GEMM does, so the error
// does not grow with K.  The tile of 256 x 16 it replaces had half the SMs idle
// and one K step of 16 in flight per block: 2^15 rows, N = 8, K = 128: 84 -> 33 us.
constexpr int kTallK = 128;
struct TallDesc {
  GemmDesc g;  // rows m in X (sa) and C (sc), columns n in W (sb) and C
  int w64;
};
template <typename TX, int NQ, int KV>
__global__ void __launch_bounds__(kSkThreads)
    k_tall(const TX* __restrict__ X, const void* __restrict__ W, float2* __restrict__ C,
           const __grid_constant__ TallDesc d) {
  constexpr int NP = 2 * NQ;
  __shared__ __align__(16) float w[kTallK * NP * 4];
  __shared__ int64_t kx[kTallK], kw[kTallK];
  __shared__ int64_t nw[4 * NQ], cn[4 * NQ];
  const GemmDesc& g = d.g;
  const int n0 = blockIdx.y * 4 * NQ, N = (int)min((int64_t)4 * NQ, g.N - n0);
  const int64_t r = (int64_t)blockIdx.x * kSkThreads + threadIdx.x;
  const bool in = r < g.M;
  if (threadIdx.x < 4 * NQ) {
    const bool col = (int)threadIdx.x < N;
    nw[threadIdx.x] = col ? offset_of(n0 + threadIdx.x, g.nn, g.ndim, g.nsb) : 0;
    cn[threadIdx.x] = col ? offset_of(n0 + threadIdx.x, g.nn, g.ndim, g.nsc) : 0;
  }
  const int64_t xr = in ? offset_of(r, g.nm, g.mdim, g.msa) : 0, cr = in ? offset_of(r, g.nm, g.mdim, g.msc) : 0;
  for (int64_t z = blockIdx.z; z < g.Z; z += gridDim.z) {
    const TX* x = X + xr + offset_of(z, g.nz, g.zdim, g.zsa);
    const int64_t zw = offset_of(z, g.nz, g.zdim, g.zsb);
    KahanC acc[4 * NQ];
#pragma unroll
    for (int n = 0; n < 4 * NQ; ++n) kahan_init(acc[n]);
    for (int64_t k0 = 0; k0 < g.K; k0 += kTallK) {
      const int kn = (int)min((int64_t)kTallK, g.K - k0), kp = (kn + 15) / 16 * 16;
      __syncthreads();  // the previous step has been read
      for (int k = threadIdx.x; k < kn; k += kSkThreads) {
        kx[k] = offset_of(k0 + k, g.nk, g.kdim, g.ksa);
        kw[k] = offset_of(k0 + k, g.nk, g.kdim, g.ksb);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < kp * 4 * NQ; t += kSkThreads) {
        const int k = t / (4 * NQ), n = t % (4 * NQ);
        float2 v = make_float2(0.f, 0.f);
        if (k < kn && n < N) {
          const int64_t o = zw + kw[k] + nw[n];
          v = d.w64 ? cvt<float>(static_cast<const double2*>(W)[o]) : static_cast<const float2*>(W)[o];
        }
        w_store(w, NP, k, n, v);
      }
      __syncthreads();
      if (!in) continue;
      for (int kc = 0; kc < kn; kc += 16) {
        TX a[16];
#pragma unroll
        for (int k = 0; k < 16; k += KV) {
          if (kc + k < kn) {
            load_run<KV>(x + kx[kc + k], &a[k]);
          } else {
#pragma unroll
            for (int u = 0; u < KV; ++u) a[k + u].x = a[k + u].y = 0;
          }
        }
        F2 ax[16], ay[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          ax[k] = f2_dup((float)a[k].x);
          ay[k] = f2_dup((float)a[k].y);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          float2 o[4];
          four_columns<16>(ax, ay, w + kc * NP * 4, NP, 4 * q, o);
#pragma unroll
          for (int n = 0; n < 4; ++n) kahan_add(acc[4 * q + n], o[n]);
        }
      }
    }
    if (in) {
      float2* c = C + cr + offset_of(z, g.nz, g.zdim, g.zsc);
#pragma unroll
      for (int n = 0; n < 4 * NQ; ++n)
        if (n < N) c[cn[n]] = kahan_value(acc[n]);
    }
  }
}

template <typename TX, int KV>
cudaError_t launch_tall_kv(const void* X, const void* W, void* C, const TallDesc& d, cudaStream_t s) {
  const int nq = d.g.N <= 4 ? 1 : 2;
  const int64_t gx = (d.g.M + kSkThreads - 1) / kSkThreads, gy = (d.g.N + 4 * nq - 1) / (4 * nq);
  if (gx > 2147483647LL || gy > 65535) return cudaErrorInvalidConfiguration;
  const dim3 grid((unsigned)gx, (unsigned)gy, (unsigned)std::min<int64_t>(d.g.Z, 65535));
  if (nq == 1)
    k_tall<TX, 1, KV><<<grid, kSkThreads, 0, s>>>((const TX*)X, W, (float2*)C, d);
  else
    k_tall<TX, 2, KV><<<grid, kSkThreads, 0, s>>>((const TX*)X, W, (float2*)C, d);
  return cudaGetLastError();
}

// Row blocks by batch index; persistent-style over the blocks that fit an SM at
// the kernels' register counts (complex64: 64 registers at K <= 16, 46 or fewer
// below; FP64: 96).
dim3 sk_grid(const SkinnyDesc& d, int per_sm, int threads = kSkThreads) {
  const int64_t y = std::min<int64_t>(d.Z, 65535);
  // (a few blocks per batch index would leave a part of the chip out or over:
  // four rounds of smaller ones; 2^15 rows, N = 1, K = 2, Z = 512: 157
  // -> 129 us)
  const int64_t fit = 152 * per_sm / y, x = std::max<int64_t>(1, fit >= 8 ? fit : 4 * 152 * per_sm / y);
  return dim3((unsigned)std::min<int64_t>((d.R + threads - 1) / threads, x), (unsigned)y);
}
// The columns, `unit` at a time, in as many groups as leave every SM four blocks
// where the rows alone do not (4096 rows, N = 128, K = 16: 43 us on 32 blocks, 11
// on 1024).
dim3 split_columns(SkinnyDesc& d, dim3 g, int unit) {
  const int units = (d.N + unit - 1) / unit;
  const int64_t want = std::max<int64_t>(1, 4 * 152 / ((int64_t)g.x * g.y));
  const int per = (int)std::max<int64_t>(1, units / std::min<int64_t>(units, want));
  d.cols = unit * per;
  g.z = (unsigned)((units + per - 1) / per);
  return g;
}

template <typename TX, typename TC, int KMAX>
cudaError_t launch_mixed_k(const void* X, const void* W, void* C, SkinnyDesc& d, int per_sm, cudaStream_t s) {
  // every block takes equally many rounds of rows, since the multiply-adds are
  // what counts (2^17.2 rows, N = 8, K = 16: 150 -> 136 us)
  const int64_t rows = (d.R + kSkThreads64 - 1) / kSkThreads64;
  dim3 grid = sk_grid(d, per_sm, kSkThreads64);
  const int64_t rounds = (rows + grid.x - 1) / grid.x;
  grid.x = (unsigned)((rows + rounds - 1) / rounds);
  // single columns where four would be padded, and where the rows are few (4096,
  // N = 4, K = 16: 14 -> 10 us)
  const bool one = d.N < 4 || (d.N < 16 && (int64_t)grid.x * grid.y <= 152);
  grid = split_columns(d, grid, one ? 1 : 4);
  const size_t smem = (size_t)KMAX * ((d.cols + 3) / 4 * 4) * (std::is_same<TC, double2>::value ? 16 : 8);
  if (one)
    k_skinny<TX, TC, KMAX, true><<<grid, kSkThreads64, smem, s>>>((const TX*)X, W, (TC*)C, d);
  else
    k_skinny<TX, TC, KMAX, false><<<grid, kSkThreads64, smem, s>>>((const TX*)X, W, (TC*)C, d);
  return cudaGetLastError();
}
template <typename TX, typename TC>
cudaError_t launch_mixed(const void* X, const void* W, void* C, SkinnyDesc& d, cudaStream_t s) {
  return d.K <= 4 ? launch_mixed_k<TX, TC, 4>(X, W, C, d, 18, s) : launch_mixed_k<TX, TC, 16>(X, W, C, d, 9, s);
}

template <int KMAX, int KV>
cudaError_t launch_kv(const void* X, const void* W, void* C, SkinnyDesc& d, cudaStream_t s) {
  dim3 grid = sk_grid(d, KMAX == 16 ? 8 : 10);
  if (d.N <= 16 && d.Z == 1 && !d.cvec) {
    k_skinny_f<KMAX, KV><<<grid, kSkThreads, 0, s>>>((const float2*)X, W, (float2*)C, d);
  } else {
    grid = split_columns(d, grid, 4);
    const size_t smem = (size_t)KMAX * (d.cols / 2) * 16;
    k_skinny_w<KMAX, KV><<<grid, kSkThreads, smem, s>>>((const float2*)X, W, (float2*)C, d);
  }
  return cudaGetLastError();
}
template <int KMAX>
cudaError_t launch_k(int kv, const void* X, const void* W, void* C, SkinnyDesc& d, cudaStream_t s) {
  if (kv == 4) return launch_kv<KMAX, 4>(X, W, C, d, s);
  if (kv == 2) return launch_kv<KMAX, 2>(X, W, C, d, s);
  return launch_kv<KMAX, 1>(X, W, C, d, s);
}

int log2_exact(int64_t v) {
  int l = 0;
  while ((int64_t(1) << l) < v) ++l;
  return (int64_t(1) << l) == v ? l : -1;
}

}  // namespace

static bool skinny_shape(const GemmDesc& g) {
  const int64_t rows = std::max(g.M, g.N);
  return rows >= kSkThreads && rows * g.Z >= kSkinnyMinRows && std::min(g.M, g.N) <= kSkinnyN && g.K <= kSkinnyK;
}

bool skinny_eligible(int precision, const GemmDesc& g) {
  if (precision == PQ_PREC_C128 && (g.Z > 1 || std::min(g.M, g.N) > kSkinnyN64)) return false;
  return skinny_shape(g);
}

cudaError_t launch_skinny(int ta, int tb, int tc, const void* A, const void* B, void* C, const GemmDesc& g,
                          cudaStream_t stream) {
  if (!skinny_shape(g)) return cudaErrorInvalidValue;
  // the large side is X (rows), the small side W
  const bool a_big = g.M >= g.N;
  const void* X = a_big ? A : B;
  const void* W = a_big ? B : A;
  const bool x64 = (a_big ? ta : tb) == PQ_C128, c64 = tc == PQ_C128;
  SkinnyDesc d;
  std::memset(&d, 0, sizeof(d));
  d.R = a_big ? g.M : g.N;
  d.Z = g.Z;
  d.N = (int)(a_big ? g.N : g.M);
  d.K = (int)g.K;
  d.w64 = (a_big ? tb : ta) == PQ_C128;
  if (d.R * d.Z == 0) return cudaSuccess;
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
  const int64_t* nsc = a_big ? g.nsc : g.msc;
  const int64_t* ndim = a_big ? g.ndim : g.mdim;
  const int nn = a_big ? g.nn : g.nm;
  bool cvec = nn > 0 && nsc[0] == 1 && ndim[0] % 4 == 0 && (uintptr_t)C % 32 == 0;
  for (int i = 1; i < nn; ++i) cvec = cvec && nsc[i] % 4 == 0;
  for (int i = 0; i < d.nr; ++i) cvec = cvec && d.rsc[i] % 4 == 0;
  d.nz = g.nz;
  for (int i = 0; i < g.nz; ++i) {
    d.zdim[i] = g.zdim[i];
    d.zsx[i] = a_big ? g.zsa[i] : g.zsb[i];
    d.zsw[i] = a_big ? g.zsb[i] : g.zsa[i];
    d.zsc[i] = g.zsc[i];
    limit(d.zsx[i]);
    cvec = cvec && d.zsc[i] % 4 == 0;
  }
  d.cvec = cvec;
  for (int k = 0; k < d.K; ++k) {
    d.kx[k] = offset_of(k, g.nk, g.kdim, ksx);
    d.kw[k] = offset_of(k, g.nk, g.kdim, a_big ? g.ksb : g.ksa);
  }
  for (int n = 0; n < d.N; ++n) {
    d.nw[n] = offset_of(n, nn, ndim, a_big ? g.nsb : g.msa);
    d.cn[n] = offset_of(n, nn, ndim, nsc);
  }
  if (c64) return x64 ? launch_mixed<double2, double2>(X, W, C, d, stream) : launch_mixed<float2, double2>(X, W, C, d, stream);
  if (x64) return launch_mixed<double2, float2>(X, W, C, d, stream);
  if (d.K <= 4) return launch_k<4>(kv, X, W, C, d, stream);
  if (d.K <= 8) return launch_k<8>(kv, X, W, C, d, stream);
  return launch_k<16>(kv, X, W, C, d, stream);
}

cudaError_t launch_tall(int ta, int tb, const void* A, const void* B, void* C, const GemmDesc& g, cudaStream_t stream) {
  TallDesc d;
  d.g = g;
  const bool a_big = g.M >= g.N;
  if (!a_big) {
    std::swap(d.g.M, d.g.N);
    std::swap(d.g.nm, d.g.nn);
    for (int i = 0; i < kMaxModes; ++i) {
      d.g.mdim[i] = g.ndim[i];
      d.g.msa[i] = g.nsb[i];
      d.g.msc[i] = g.nsc[i];
      d.g.ndim[i] = g.mdim[i];
      d.g.nsb[i] = g.msa[i];
      d.g.nsc[i] = g.msc[i];
      std::swap(d.g.ksa[i], d.g.ksb[i]);
      std::swap(d.g.zsa[i], d.g.zsb[i]);
    }
    std::swap(A, B);
    std::swap(ta, tb);
  }
  d.w64 = tb == PQ_C128;
  if (d.g.M * d.g.N * d.g.Z == 0) return cudaSuccess;
  if (ta == PQ_C128) return launch_tall_kv<double2, 1>(A, B, C, d, stream);
  // aligned runs along K, as for the skinny pairs
  int kv = d.g.nk > 0 && d.g.ksa[0] == 1 ? 4 : 1;
  auto limit = [&](int64_t v) {
    while (kv > 1 && v % kv) kv /= 2;
  };
  if (kv > 1) limit(d.g.kdim[0]);
  while (kv > 1 && (uintptr_t)A % (8 * kv)) kv /= 2;
  for (int i = 1; i < d.g.nk; ++i) limit(d.g.ksa[i]);
  for (int i = 0; i < d.g.nm; ++i) limit(d.g.msa[i]);
  for (int i = 0; i < d.g.nz; ++i) limit(d.g.zsa[i]);
  if (kv == 4) return launch_tall_kv<float2, 4>(A, B, C, d, stream);
  if (kv == 2) return launch_tall_kv<float2, 2>(A, B, C, d, stream);
  return launch_tall_kv<float2, 1>(A, B, C, d, stream);
}

}  // namespace pq
