// Inline-PTX building blocks shared by the tcgen05 kernels (pq_tc.cu,
// pq_oz.cu): mbarriers with bounded waits, 1D bulk copies into shared memory,
// UMMA shared-memory / instruction descriptors, tcgen05.mma issue and commit,
// TMEM loads and fences, and the host-side SM count for persistent grids.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pq_internal.h"
#include "pq_types.cuh"

namespace pq {
namespace tcg {

constexpr uint32_t kWaitLimit = 1u << 22;  // mbarrier polls before giving up
constexpr int kStatusTcTimeout = 0x7c01;   // status word value after a wait expired

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Offset of linear index x over n mixed-radix modes with strides s1.
__device__ __forceinline__ int64_t decode(int64_t x, int n, const int64_t* dim, const int64_t* s1) {
  int64_t o = 0;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    int64_t q = x / dim[i];
    o += (x - q * dim[i]) * s1[i];
    x = q;
  }
  return o;
}

// The same in 32-bit steps, a shift where the extent is a power of two, for the
// passes that decode an index per element or per row (a 64-bit division costs
// some 70 instructions); indices of 2^32 and more take decode().  In the index
// table, packs and exponent passes: 5x6 depth-14 amplitudes in 3xTF32 8.55 -> 8.43
// ms, 64 amplitudes of 5x5 depth 14 3.67 -> 3.63 ms.  The exact-accumulation
// GEMM's converters keep decode(): 1 % slower with this on operands stored along M.
__device__ __forceinline__ int64_t decode32(int64_t x, int n, const int64_t* dim, const int64_t* s1) {
  if ((uint64_t)x >> 32) return decode(x, n, dim, s1);
  int64_t o = 0;
  uint32_t y = (uint32_t)x;
#pragma unroll 1
  for (int i = 0; i < n; ++i) {
    const int64_t dm = dim[i];
    uint32_t q = 0, r = y;
    if (!((uint64_t)dm >> 32)) {
      const uint32_t d = (uint32_t)dm;
      if ((d & (d - 1)) == 0) {
        q = y >> (__ffs((int)d) - 1);
        r = y & (d - 1);
      } else {
        q = y / d;
        r = y - q * d;
      }
    }
    o += (int64_t)r * s1[i];
    y = q;
  }
  return o;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait for the phase of the given parity: at most `limit` polls;
// false when it expired.
__device__ __forceinline__ bool mbar_wait_polls(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  return mbar_wait_polls(bar, parity, kWaitLimit);
}
// Records an expired wait in the context's status word (read by the host at
// the next synchronising call, where it becomes PQ_ERR_DEVICE).
__device__ __forceinline__ void report_timeout(int* status) {
  if (status) atomicExch_system(status, kStatusTcTimeout);
}
// 1D bulk copy global -> shared (16-byte aligned addresses, size a multiple
// of 16), completing as transaction bytes on `bar`.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Shared-memory matrix descriptor from an address in 16-byte units: no
// swizzle, K-major canonical layout (8-row x 16-byte core matrices; lbo =
// K-adjacent core stride, sbo = 8-row-group stride, both in bytes), descriptor
// version 1 (sm_100-family tcgen05) in bit 46.
__device__ __forceinline__ uint64_t desc_at(uint32_t addr16, uint32_t lbo, uint32_t sbo) {
  const uint32_t lo = addr16 | (lbo >> 4) << 16, hi = (sbo >> 4) | 1u << 14;
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
// One thread of a converged warp (the same one every time).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e != 0;
}
// Instruction descriptors, FP32 accumulation, both operands K-major; bit 13
// negates A.  kind::tf32: A/B format 2; kind::f16: 0 for fp16 operands, 1 for
// bf16 (both operands of one MMA alike).
__host__ __device__ constexpr uint32_t idesc_tf32(int m, int n, bool neg_a = false) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((neg_a ? 1u : 0u) << 13) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
__host__ __device__ constexpr uint32_t idesc_f16(bool half, int m, int n, bool neg_a = false) {
  return (1u << 4) | ((half ? 0u : 1u) << 7) | ((half ? 0u : 1u) << 10) | ((neg_a ? 1u : 0u) << 13) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// The same MMA for consecutive ones with the same A operand: the first keeps A
// in the tensor core's buffer (fill), the others take it from there, the last
// for the last time.
__device__ __forceinline__ void mma_f16_a_fill(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_f16_a_use(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16.collector::a::use [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_f16_a_lastuse(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// Arrives on `bar` once every tcgen05 operation issued so far by this thread
// has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Stores 16 consecutive 32-bit columns of the warp's 32 TMEM lanes (one
// value per lane and column), the inverse of tmem_ld16.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Result offsets of every row (m) and column (n) of C, decoded once per
// launch (a template so that each translation unit may instantiate it).
template <int Unused = 0>
__global__ void __launch_bounds__(256) k_result_index(const __grid_constant__ GemmDesc d, int64_t* __restrict__ cm,
                                                      int64_t* __restrict__ cn) {
  pdl_trigger();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < d.M + d.N; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t o = i < d.M ? decode32(i, d.nm, d.mdim, d.msc) : decode32(i - d.M, d.nn, d.ndim, d.nsc);
    pdl_wait();  // the tables may still be read by the launch before
    if (i < d.M)
      cm[i] = o;
    else
      cn[i - d.M] = o;
  }
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// SMs of the current device (cached per device), the persistent grid size.
inline int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 1;
    cached[dev] = n;
  }
  return cached[dev];
}

}  // namespace tcg
}  // namespace pq
