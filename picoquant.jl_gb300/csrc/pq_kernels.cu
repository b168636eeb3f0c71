// SIMT kernels for sm_103a: the fused permute+contract kernel for
// memory-bound pairs, and data movement (permute/view, gather, slice gather,
// FP64 compensated slice sum).
//
// Every operand and the result carry their own storage type (complex64 or
// complex128).  Results stored as complex128 are accumulated in FP64; results
// stored as complex64 are accumulated in FP32 over chunks of kChunk terms that
// are folded with Kahan compensation.
#include <algorithm>

#include "pq_types.cuh"

namespace pq {

// Decode linear index `c` over the result modes into offsets in A and B.
template <bool POW2>
__device__ __forceinline__ void decode2(int64_t c, const GenericDesc& d, int64_t& oa, int64_t& ob) {
  oa = 0;
  ob = 0;
#pragma unroll 1
  for (int i = 0; i < d.nc; ++i) {
    int64_t r;
    if (POW2) {
      r = c & (d.cdim[i] - 1);
      c >>= d.clog[i];
    } else {
      int64_t q = c / d.cdim[i];
      r = c - q * d.cdim[i];
      c = q;
    }
    oa += r * d.csa[i];
    ob += r * d.csb[i];
  }
}

template <bool POW2>
__device__ __forceinline__ void decodek(int64_t k, const GenericDesc& d, int64_t& oa, int64_t& ob) {
  oa = 0;
  ob = 0;
#pragma unroll 1
  for (int i = 0; i < d.nk; ++i) {
    int64_t r;
    if (POW2) {
      r = k & (d.kdim[i] - 1);
      k >>= d.klog[i];
    } else {
      int64_t q = k / d.kdim[i];
      r = k - q * d.kdim[i];
      k = q;
    }
    oa += r * d.ksa[i];
    ob += r * d.ksb[i];
  }
}

constexpr int kGenThreads = 256;

// Sum over k of A[a + ka[k]] * B[b + kb[k]] for k in [0, kn): every L-th term
// from sub, accumulated into `acc` (FP64), or all terms into the compensated
// accumulator (FP32).
template <typename TA, typename TB>
__device__ __forceinline__ void dot_chunk(double2& acc, KahanC&, const TA* a, const TB* b, const int64_t* ka,
                                          const int64_t* kb, int kn, int sub, int L) {
#pragma unroll 4
  for (int k = sub; k < kn; k += L) cfma(acc, cvt<double>(a[ka[k]]), cvt<double>(b[kb[k]]));
}
template <typename TA, typename TB>
__device__ __forceinline__ void dot_chunk(float2&, KahanC& ks, const TA* a, const TB* b, const int64_t* ka,
                                          const int64_t* kb, int kn, int, int) {
  int k = 0;
  for (; k + kChunk <= kn; k += kChunk) {
    float2 p = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < kChunk; ++j) cfma(p, cvt<float>(a[ka[k + j]]), cvt<float>(b[kb[k + j]]));
    kahan_add(ks, p);
  }
  float2 p = make_float2(0.f, 0.f);
  for (; k < kn; ++k) cfma(p, cvt<float>(a[ka[k]]), cvt<float>(b[kb[k]]));
  kahan_add(ks, p);
}

__device__ __forceinline__ double2 acc_value(const double2& acc, const KahanC&) { return acc; }
__device__ __forceinline__ float2 acc_value(const float2&, const KahanC& ks) { return kahan_value(ks); }

// Partial sums of the 2^lsub consecutive lanes that share a result element
// (every lane of the warp takes part).
__device__ __forceinline__ void fold_lanes(double2& acc, int lsub) {
  for (int o = (1 << lsub) >> 1; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
}
__device__ __forceinline__ void fold_lanes(float2&, int) {}

// Lanes (2^l) per result element of an FP64 contraction.  A small result leaves
// most of the chip idle while each thread walks its K terms in sequence (FP64
// multiply-adds and cached loads, about 30 ns per term): K is shared by up to 32
// lanes while all threads fit the chip about once and each keeps four terms.
// 1 x 512 terms: 17 -> 5 us.
int generic_lanes(int64_t csize, int64_t ksize) {
  int l = 0;
  while (l < 5 && (csize << (l + 1)) <= 152 * 1024 && (ksize >> (l + 1)) >= 4) ++l;
  return l;
}

template <typename TA, typename TB, typename TC, typename R, bool POW2>
__global__ void __launch_bounds__(kGenThreads)
    k_generic(const TA* A, const TB* B, TC* C,
              const __grid_constant__ GenericDesc d, int lsub) {
  __shared__ int64_t ka[kGenericKTab];
  __shared__ int64_t kb[kGenericKTab];
  using AC = typename Acc<R>::C;
  const int64_t K = d.ksize;
  const int KT = (int)(K < kGenericKTab ? K : kGenericKTab);
  const bool one_chunk = K <= kGenericKTab;
  if (one_chunk) {
    for (int k = threadIdx.x; k < KT; k += blockDim.x) {
      int64_t x, y;
      decodek<POW2>(k, d, x, y);
      ka[k] = x;
      kb[k] = y;
    }
    __syncthreads();
  }
  pdl_wait();
  // Up to two blocks per SM the launch after may start beside this one (5 % of
  // back-to-back launches).  Blocks of a larger one would be placed where this
  // one has left room, unevenly over the SMs, and then run there: 2^17 results,
  // K = 64, one launch after the other: 88 us each so, 67 without; 3 to 7 blocks
  // per SM 16 % in the mean.
  if (gridDim.x <= 304) pdl_trigger();
  const int L = 1 << lsub;
  const int64_t total = d.csize << lsub;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < total; base += step) {
    const int64_t c = (base + threadIdx.x) >> lsub;
    const int sub = threadIdx.x & (L - 1);
    const bool active = c < d.csize;
    int64_t oa = 0, ob = 0;
    if (active) decode2<POW2>(c, d, oa, ob);
    AC acc = czero(R());
    KahanC ks;
    kahan_init(ks);
    if (one_chunk) {
      if (active) dot_chunk(acc, ks, A + oa, B + ob, ka, kb, KT, sub, L);
    } else {
      for (int64_t k0 = 0; k0 < K; k0 += KT) {
        const int kn = (int)((K - k0) < KT ? (K - k0) : KT);
        __syncthreads();
        for (int k = threadIdx.x; k < kn; k += blockDim.x) {
          int64_t x, y;
          decodek<POW2>(k0 + k, d, x, y);
          ka[k] = x;
          kb[k] = y;
        }
        __syncthreads();
        if (active) dot_chunk(acc, ks, A + oa, B + ob, ka, kb, kn, sub, L);
      }
    }
    fold_lanes(acc, lsub);
    if (active && sub == 0) C[c] = store_as<TC>(acc_value(acc, ks));
  }
}

template <typename TA, typename TB, typename TC>
static cudaError_t gen_launch(const void* A, const void* B, void* C, const GenericDesc& d, cudaStream_t s) {
  using R = typename std::conditional<std::is_same<TC, double2>::value, double, float>::type;
  const int l = std::is_same<TC, double2>::value ? generic_lanes(d.csize, d.ksize) : 0;
  const dim3 grid((unsigned)grid_for(d.csize << l, kGenThreads)), block(kGenThreads);
  return d.pow2 ? launch_pdl(k_generic<TA, TB, TC, R, true>, grid, block, 0, s, (const TA*)A, (const TB*)B, (TC*)C, d, l)
                : launch_pdl(k_generic<TA, TB, TC, R, false>, grid, block, 0, s, (const TA*)A, (const TB*)B, (TC*)C, d, l);
}

template <typename TA, typename TB>
static cudaError_t gen_launch_c(int tc, const void* A, const void* B, void* C, const GenericDesc& d, cudaStream_t s) {
  return tc == PQ_C128 ? gen_launch<TA, TB, double2>(A, B, C, d, s) : gen_launch<TA, TB, float2>(A, B, C, d, s);
}

cudaError_t launch_generic(int ta, int tb, int tc, const void* A, const void* B, void* C, const GenericDesc& d,
                           cudaStream_t stream) {
  if (d.csize == 0) return cudaSuccess;
  if (ta == PQ_C128 && tb == PQ_C128) return gen_launch_c<double2, double2>(tc, A, B, C, d, stream);
  if (ta == PQ_C128) return gen_launch_c<double2, float2>(tc, A, B, C, d, stream);
  if (tb == PQ_C128) return gen_launch_c<float2, double2>(tc, A, B, C, d, stream);
  return gen_launch_c<float2, float2>(tc, A, B, C, d, stream);
}

// Grouped small steps: one launch runs up to kGroupMax independent small
// contractions (complex128 operands and results, K <= kGroupK), each on its
// own range of blocks.  A block finds its member in the prefix table, copies
// the member's descriptor (prepared once per plan) into shared memory and
// runs the generic kernel's loop on it.  Everything before pdl_wait() reads
// tables that no kernel writes, so it overlaps the launch before.
__global__ void __launch_bounds__(kGenThreads)
    k_generic_group(const __grid_constant__ GenericGroup g, const GenericDesc* __restrict__ descs) {
  __shared__ GenericDesc sd;
  __shared__ int64_t ka[kGroupK];
  __shared__ int64_t kb[kGroupK];
  int m = 0;
  while (m + 1 < g.n && g.blk[m + 1] <= (int)blockIdx.x) ++m;
  {
    const int* src = reinterpret_cast<const int*>(descs + g.desc[m]);
    int* dst = reinterpret_cast<int*>(&sd);
    for (int t = threadIdx.x; t < (int)(sizeof(GenericDesc) / sizeof(int)); t += blockDim.x) dst[t] = src[t];
  }
  __syncthreads();
  const int KT = (int)sd.ksize;
  for (int k = threadIdx.x; k < KT; k += blockDim.x) {
    int64_t x, y;
    if (sd.pow2)
      decodek<true>(k, sd, x, y);
    else
      decodek<false>(k, sd, x, y);
    ka[k] = x;
    kb[k] = y;
  }
  __syncthreads();
  const double2* A = static_cast<const double2*>(g.A[m]);
  const double2* B = static_cast<const double2*>(g.B[m]);
  double2* C = static_cast<double2*>(g.C[m]);
  const int lsub = g.lsub[m], L = 1 << lsub;
  const int64_t nb = g.blk[m + 1] - g.blk[m];
  const int64_t step = nb * blockDim.x, total = sd.csize << lsub;
  pdl_wait();
  pdl_trigger();
  for (int64_t base = (int64_t)(blockIdx.x - g.blk[m]) * blockDim.x; base < total; base += step) {
    const int64_t c = (base + threadIdx.x) >> lsub;
    const int sub = threadIdx.x & (L - 1);
    const bool active = c < sd.csize;
    double2 acc = make_double2(0.0, 0.0);
    KahanC ks;
    if (active) {
      int64_t oa, ob;
      if (sd.pow2)
        decode2<true>(c, sd, oa, ob);
      else
        decode2<false>(c, sd, oa, ob);
      dot_chunk(acc, ks, A + oa, B + ob, ka, kb, KT, sub, L);
    }
    fold_lanes(acc, lsub);
    if (active && sub == 0) C[c] = acc;
  }
}

cudaError_t launch_generic_group(const GenericGroup& g, const GenericDesc* d_descs, cudaStream_t stream) {
  if (g.n <= 0 || g.blk[g.n] <= 0) return cudaSuccess;
  return launch_pdl(k_generic_group, dim3((unsigned)g.blk[g.n]), dim3(kGenThreads), 0, stream, g, d_descs);
}

// ---------------------------------------------------------------------------
// Data movement
// ---------------------------------------------------------------------------
template <typename TI, typename TO, bool POW2>
__global__ void __launch_bounds__(kGenThreads)
    k_permute(const TI* __restrict__ in, int64_t base, TO* __restrict__ out, const __grid_constant__ GenericDesc d) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < d.csize; c += step) {
    int64_t oa, ob;
    decode2<POW2>(c, d, oa, ob);
    out[c] = store_as<TO>(in[base + oa]);
  }
}

template <typename TI, typename TO>
static void perm_launch(const void* in, int64_t base, void* out, const GenericDesc& d, cudaStream_t s) {
  const int grid = grid_for(d.csize, kGenThreads);
  if (d.pow2)
    k_permute<TI, TO, true><<<grid, kGenThreads, 0, s>>>((const TI*)in, base, (TO*)out, d);
  else
    k_permute<TI, TO, false><<<grid, kGenThreads, 0, s>>>((const TI*)in, base, (TO*)out, d);
}

cudaError_t launch_permute(int tin, int tout, const void* in, int64_t base, void* out, const GenericDesc& d,
                           cudaStream_t stream) {
  if (d.csize == 0) return cudaSuccess;
  if (tin == PQ_C128) {
    if (tout == PQ_C128)
      perm_launch<double2, double2>(in, base, out, d, stream);
    else
      perm_launch<double2, float2>(in, base, out, d, stream);
  } else {
    if (tout == PQ_C128)
      perm_launch<float2, double2>(in, base, out, d, stream);
    else
      perm_launch<float2, float2>(in, base, out, d, stream);
  }
  return cudaGetLastError();
}

template <typename T>
__global__ void k_gather(const T* __restrict__ in, const int64_t* __restrict__ idx, int64_t n, T* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[idx[i]];
}

cudaError_t launch_gather(int dt, const void* in, const int64_t* d_idx, int64_t n, void* out, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  int grid = (int)((n + 255) / 256);
  if (dt == PQ_C128)
    k_gather<double2><<<grid, 256, 0, stream>>>((const double2*)in, d_idx, n, (double2*)out);
  else
    k_gather<float2><<<grid, 256, 0, stream>>>((const float2*)in, d_idx, n, (float2*)out);
  return cudaGetLastError();
}

// One block per job (grid-stride over jobs): 16-byte vector copies, an
// 8-byte tail by thread 0.
__global__ void __launch_bounds__(256) k_scatter(const unsigned char* __restrict__ src,
                                                 const CopyJob* __restrict__ jobs, int n) {
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    const CopyJob cj = jobs[j];
    const uint4* s = reinterpret_cast<const uint4*>(src + cj.src_off);
    uint4* d = reinterpret_cast<uint4*>(cj.dst);
    const int64_t n16 = cj.bytes / 16;
    for (int64_t i = threadIdx.x; i < n16; i += blockDim.x) d[i] = s[i];
    if (threadIdx.x == 0 && (cj.bytes & 15))
      reinterpret_cast<uint2*>(cj.dst)[2 * n16] = reinterpret_cast<const uint2*>(src + cj.src_off)[2 * n16];
  }
}

cudaError_t launch_scatter(const void* src, const CopyJob* d_jobs, int n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int grid = n < 152 * 8 ? n : 152 * 8;
  k_scatter<<<grid, 256, 0, stream>>>((const unsigned char*)src, d_jobs, n);
  return cudaGetLastError();
}

template <typename T>
__device__ __forceinline__ void slice_copy(const T* in, T* out, const SliceJob& j, int64_t first, int64_t step,
                                           int64_t s0, int64_t nb, int64_t s_end) {
  const int64_t total = j.d.csize * nb;
  for (int64_t e = first; e < total; e += step) {
    int64_t b = e / j.d.csize;
    int64_t x = e - b * j.d.csize;
    int64_t s = s0 + b, so = 0;
    if (s >= s_end) {
      out[e] = T{0, 0};
      continue;
    }
    for (int i = 0; i < j.nsl; ++i) {
      int64_t q = s / j.dim[i];
      so += (s - q * j.dim[i]) * j.stride[i];
      s = q;
    }
    int64_t oa, ob;
    decode2<false>(x, j.d, oa, ob);
    out[e] = in[so + oa];
  }
}

// The sliced leaves of one batch in one launch (one launch each took 12 of the
// 67 launches of a small sliced amplitude): a block finds its leaf in the prefix
// table and copies that leaf's descriptor into shared memory while the launch
// before still runs.
__global__ void __launch_bounds__(kGenThreads)
    k_slice_gather(const __grid_constant__ SliceGroup g, const SliceJob* __restrict__ jobs, int64_t s0, int64_t nb,
                   int64_t s_end) {
  __shared__ SliceJob job;
  int m = 0;
  while (m + 1 < g.n && g.blk[m + 1] <= (int)blockIdx.x) ++m;
  const int* src = reinterpret_cast<const int*>(jobs + g.job0 + m);
  for (int t = threadIdx.x; t < (int)(sizeof(SliceJob) / sizeof(int)); t += blockDim.x)
    reinterpret_cast<int*>(&job)[t] = src[t];
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const int64_t step = (int64_t)(g.blk[m + 1] - g.blk[m]) * blockDim.x;
  const int64_t first = (int64_t)(blockIdx.x - g.blk[m]) * blockDim.x + threadIdx.x;
  if (job.dt == PQ_C128)
    slice_copy(static_cast<const double2*>(g.in[m]), static_cast<double2*>(g.out[m]), job, first, step, s0, nb, s_end);
  else
    slice_copy(static_cast<const float2*>(g.in[m]), static_cast<float2*>(g.out[m]), job, first, step, s0, nb, s_end);
}

cudaError_t launch_slice_gather(const SliceGroup& g, const SliceJob* d_jobs, int64_t s0, int64_t nb, int64_t s_end,
                                cudaStream_t stream) {
  if (g.n <= 0 || g.blk[g.n] <= 0) return cudaSuccess;
  return launch_pdl(k_slice_gather, dim3((unsigned)g.blk[g.n]), dim3(kGenThreads), 0, stream, g, d_jobs, s0, nb, s_end);
}

// Neumaier compensated accumulation of one value into (s, c).
__device__ __forceinline__ void neumaier(double& s, double& c, double x) {
  double t = s + x;
  if (fabs(s) >= fabs(x))
    c += (s - t) + x;
  else
    c += (x - t) + s;
  s = t;
}

// One warp per element: lanes accumulate strided subsets of the batch, then the
// 32 partial (sum, compensation) pairs are folded pairwise (lane l takes lane
// l + o, o = 16 .. 1), so the result is deterministic: five dependent steps
// instead of the 32 of a fold by one lane (21 -> 9 us for 64 slices).
template <typename T>
__global__ void k_slice_sum(const T* X, int64_t n, int64_t nb, double* acc, double* comp) {
  const int lane = threadIdx.x & 31;
  const int64_t e = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  pdl_wait();
  pdl_trigger();
  if (e >= n) return;
  double sr = 0, cr = 0, si = 0, ci = 0;
  for (int64_t b = lane; b < nb; b += 32) {
    T v = X[e + n * b];
    neumaier(sr, cr, (double)v.x);
    neumaier(si, ci, (double)v.y);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double a = __shfl_down_sync(0xffffffffu, sr, o), b = __shfl_down_sync(0xffffffffu, cr, o);
    const double c = __shfl_down_sync(0xffffffffu, si, o), dd = __shfl_down_sync(0xffffffffu, ci, o);
    neumaier(sr, cr, a);
    cr += b;
    neumaier(si, ci, c);
    ci += dd;
  }
  if (lane == 0) {
    double r_s = acc[2 * e], r_c = comp[2 * e], i_s = acc[2 * e + 1], i_c = comp[2 * e + 1];
    neumaier(r_s, r_c, sr);
    neumaier(i_s, i_c, si);
    acc[2 * e] = r_s;
    comp[2 * e] = r_c + cr;
    acc[2 * e + 1] = i_s;
    comp[2 * e + 1] = i_c + ci;
  }
}

// Squared 2-norm of a complex tensor in FP64 (the fidelity check of a state
// vector): pass 1, every thread a Neumaier sum of |x|^2 over a grid-stride
// range, the block's sums folded by one thread in a fixed order into
// part[block] (value, compensation); pass 2, one thread folds the blocks' parts
// in block order.  Deterministic: no atomics.
constexpr int kNormThreads = 256;
template <typename T>
__global__ void __launch_bounds__(kNormThreads) k_norm2(const T* __restrict__ X, int64_t n, double* part) {
  __shared__ double ss[kNormThreads], sc[kNormThreads];
  double s = 0, c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T v = X[i];
    neumaier(s, c, (double)v.x * (double)v.x);
    neumaier(s, c, (double)v.y * (double)v.y);
  }
  ss[threadIdx.x] = s;
  sc[threadIdx.x] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    double bs = 0, bc = 0;
    for (int t = 0; t < (int)blockDim.x; ++t) {
      neumaier(bs, bc, ss[t]);
      bc += sc[t];
    }
    part[2 * blockIdx.x] = bs;
    part[2 * blockIdx.x + 1] = bc;
  }
}
__global__ void k_norm2_fold(const double* __restrict__ part, int nblocks, double* out) {
  if (threadIdx.x != 0) return;
  double s = 0, c = 0;
  for (int b = 0; b < nblocks; ++b) {
    neumaier(s, c, part[2 * b]);
    c += part[2 * b + 1];
  }
  *out = s + c;
}

int norm2_blocks(int64_t n) { return (int)std::min<int64_t>(std::max<int64_t>((n + kNormThreads - 1) / kNormThreads, 1), 1024); }

cudaError_t launch_norm2(int dt, const void* X, int64_t n, double* part, double* out, cudaStream_t stream) {
  const int nb = norm2_blocks(n);
  if (dt == PQ_C128)
    k_norm2<double2><<<nb, kNormThreads, 0, stream>>>((const double2*)X, n, part);
  else
    k_norm2<float2><<<nb, kNormThreads, 0, stream>>>((const float2*)X, n, part);
  k_norm2_fold<<<1, 32, 0, stream>>>(part, nb, out);
  return cudaGetLastError();
}

cudaError_t launch_slice_sum(int dt, const void* X, int64_t n, int64_t nb, double* acc, double* comp,
                             cudaStream_t stream) {
  if (n == 0 || nb == 0) return cudaSuccess;
  const int warps = 4;
  int grid = (int)((n + warps - 1) / warps);
  if (dt == PQ_C128)
    return launch_pdl(k_slice_sum<double2>, dim3(grid), dim3(32 * warps), 0, stream, (const double2*)X, n, nb, acc, comp);
  return launch_pdl(k_slice_sum<float2>, dim3(grid), dim3(32 * warps), 0, stream, (const float2*)X, n, nb, acc, comp);
}

}  // namespace pq
