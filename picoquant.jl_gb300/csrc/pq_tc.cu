// Split-precision complex contraction on the 5th-generation tensor cores
// (tcgen05, sm_103a): TF32 split products, FP32 accumulation in TMEM over
// 16-deep K chunks, chunk sums folded into Kahan-compensated FP32 registers.
//
//   C = A x B (complex), two real accumulators per output tile
//     Cr = Ar.Br + (-Ai).Bi   (the negation is the MMA's negate-A bit)
//     Ci = Ar.Bi + Ai.Br
//   Every real value is split into NS TF32 terms x = x0 + x1 (+ x2), each the
//   round-to-nearest TF32 value of the remainder, and a real product is the
//   sum of the term products with i + j < NS:
//     NS = 2 (PQ_PREC_3XTF32): x0y0 + x0y1 + x1y0                (3 products)
//     NS = 3 (PQ_PREC_6XTF32): x0y0 + x0y1 + x1y0 + x0y2 + x2y0 + x1y1  (6)
//
// k_tc_pack gathers an operand through its index map (any mode order, batch
// modes) into the terms of its real and imaginary parts, laid out tile by tile;
// a tile is ROWS (128 for A, 64 for B) x 16 K values in the canonical
// no-swizzle K-major UMMA layout: 8-row x 16-byte core matrices (128 contiguous
// bytes), row-adjacent core matrices 128 bytes apart.  A has one plane per part
// and term; B one plane per term, of 128 rows: the 64 of the real part, then the
// 64 of the imaginary part, so that Ar.[Br Bi] is one MMA.  Rows and K beyond
// the operand are zero.
//
// k_tc_gemm: one CTA per 128 x 64 output tile (x batch), 18 warps.
//   warp 0   producer: two cp.async.bulk per 16-deep K tile (the A and the B
//            planes, each contiguous) into a shared-memory ring (mbarrier
//            complete_tx);
//   warp 1   allocates TMEM and issues tcgen05.mma (M=128, K=8); every 16-deep
//            K tile is one chunk, rotating over four sets of two 64-column FP32
//            accumulators (all 512 TMEM columns), committed to the epilogue per
//            chunk;
//   warps 2-17 epilogue: warp w reads TMEM lanes 32*(w%4).. and 16 of the 64
//            columns, folds each chunk's (Cr, Ci) into Kahan sums (two columns
//            per f32x2 instruction), hands the accumulator set back, and finally
//            scatters C through the result index map.
// What bounds it: the MMAs (about 1500 SM cycles per K tile with two terms) and
// the epilogue (1400) are close to each other, the bulk copies need 900 (each
// measured with the others' work left out; 1600 together).  With both packs, the
// index table and the launches, 8192 x 512 x 1024 (M x N x K) takes 235 us (300
// with N = 64 MMAs and scalar sums) and 32768 x 128 x 128 takes 60 us; 128 x 48
// tiles, which read A three times for N = 128 and pad it to 144, and packs of
// one value per thread took 52 us for its GEMM and 27 (now 17) for A's pack alone.
// The four launches of a pair are programmatic dependents of each other, so that
// index decodes and barrier set-up run while the launch before them drains.
// The tensor core rounds accumulations toward zero.  The small correction
// products of a chunk go in first, the hi x hi products last, so each chunk
// takes its few truncations at (partial) full magnitude; chunks are summed
// with compensation, which keeps the bias from growing with K, and the
// expected shrinkage of those truncations is added back in the final store.
// Every mbarrier wait is bounded; on expiry the kernel records an error in the
// context's status word and runs to the end (TMEM is always released), so the
// host sees PQ_ERR_DEVICE, not a hang.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "pq_tcgen05.cuh"
#include "pq_types.cuh"

namespace pq {

namespace {

using namespace tcg;

constexpr int TM = 128, TN = 64, TK = 16;
constexpr int kThreads = 576;                  // producer, MMA, 16 epilogue warps
constexpr int kEpiWarps = 16;
constexpr int kSets = 4;                       // TMEM accumulator sets in rotation
constexpr uint32_t kTmemCols = 512;            // 4 sets x 2 accumulators x 64 columns
// Expected relative shrinkage of a value truncated (rounded toward zero) to
// FP32: half an ulp over a log-uniform mantissa, 2^-24 * ln 2 ...
constexpr float kTruncUnit = 4.13145e-8f;
// ... times the effective number of full-magnitude truncations per chunk: the
// four hi x hi additions into an accumulator land on partial sums of about
// 1/4, 1/2, 3/4 and all of the chunk value (random-sign terms), 2.5 in all;
// measured on random complex operands the shrinkage is 2.2 units (the
// partial sums' mantissas are not log-uniform).
constexpr float kTruncBias = 2.2f * kTruncUnit;
constexpr int kATile = TM * TK;                // floats per A plane tile (8 KiB)
constexpr int kBTile = TN * TK;                // floats per B plane tile (4 KiB)

template <int NS>
struct Cfg {
  static constexpr int planes = 2 * NS;                                  // per operand
  static constexpr uint32_t stage_bytes = planes * (kATile + kBTile) * 4;
  static constexpr int stages = NS == 2 ? 4 : 3;
  static constexpr int products = NS == 2 ? 3 : 6;
};

__device__ __forceinline__ float tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

template <int NS>
__device__ __forceinline__ void split(float x, float* t) {
  t[0] = tf32_rna(x);
  float r = x - t[0];
  t[1] = tf32_rna(r);
  if (NS == 3) t[2] = tf32_rna(r - t[1]);
}
template <int NS>
__device__ __forceinline__ void split(double x, float* t) {
  t[0] = tf32_rna((float)x);
  double r = x - (double)t[0];
  t[1] = tf32_rna((float)r);
  if (NS == 3) t[2] = tf32_rna((float)(r - (double)t[1]));
}

// Pack operand X (side 0: A with m modes, side 1: B with n modes) into planes
// laid out [z][row tile][k tile][plane][ROWS*16 floats].  A block packs `kper`
// K tiles of one row tile, a thread four K values of one row at a time: one
// 32-byte load where they are adjacent and aligned (four 8-byte ones where
// not), one 16-byte store per plane.  The rows' offsets (a mixed-radix decode)
// are found once per block, and before the kernel waits for the operand.
constexpr int kPackMaxK = 8;  // K tiles per block at most
template <typename T, int NS, int ROWS>
__global__ void __launch_bounds__(256) k_tc_pack(const T* X, float* planes, const __grid_constant__ GemmDesc d,
                                                 int side, int64_t rows, int64_t rtiles, int64_t ktiles, int kper) {
  constexpr int TILE = ROWS * TK, QUADS = TILE / 4;
  __shared__ int64_t roff[ROWS];
  __shared__ int64_t koff[kPackMaxK * TK];
  const int64_t kt0 = blockIdx.x * (int64_t)kper, rt = blockIdx.y, z = blockIdx.z;
  const int nkt = (int)(ktiles - kt0 < kper ? ktiles - kt0 : kper);
  const int nrm = side == 0 ? d.nm : d.nn;
  const int64_t* rdim = side == 0 ? d.mdim : d.ndim;
  const int64_t* rstr = side == 0 ? d.msa : d.nsb;
  const int64_t* kstr = side == 0 ? d.ksa : d.ksb;
  const int64_t* zstr = side == 0 ? d.zsa : d.zsb;
  for (int t = threadIdx.x; t < ROWS + nkt * TK; t += blockDim.x) {
    if (t < ROWS) {
      int64_t r = rt * ROWS + t;
      roff[t] = r < rows ? decode32(r, nrm, rdim, rstr) : -1;
    } else {
      int64_t k = kt0 * TK + (t - ROWS);
      koff[t - ROWS] = k < d.K ? decode32(k, d.nk, d.kdim, kstr) : -1;
    }
  }
  const T* Xz = X + decode32(z, d.nz, d.zdim, zstr);
  pdl_trigger();
  pdl_wait();
  __syncthreads();
  float* tiles = planes + (((z * rtiles + rt) * ktiles + kt0) * (2 * NS)) * (int64_t)TILE;
#pragma unroll 2
  for (int o = threadIdx.x; o < nkt * QUADS; o += blockDim.x) {
    // quad w of tile t: core matrix (kc, row group) row by row = kc * ROWS + row
    const int t = o / QUADS, w = o - t * QUADS, kc = w / ROWS, r = w - kc * ROWS;
    const int64_t* ko = koff + t * TK + kc * 4;
    const int64_t ro = roff[r], k0 = ko[0], k1 = ko[1], k2 = ko[2], k3 = ko[3];
    T v[4] = {};
    if (ro >= 0) {
      const T* x = Xz + ro;
      bool wide = false;
      if constexpr (sizeof(T) == 8)
        wide = k0 >= 0 && k1 == k0 + 1 && k2 == k0 + 2 && k3 == k0 + 3 && ((uintptr_t)(x + k0) & 31) == 0;
      if (wide) {
        if constexpr (sizeof(T) == 8)
          asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y),
                         "=f"(v[3].x), "=f"(v[3].y)
                       : "l"(x + k0));
      } else {
        if (k0 >= 0) v[0] = x[k0];
        if (k1 >= 0) v[1] = x[k1];
        if (k2 >= 0) v[2] = x[k2];
        if (k3 >= 0) v[3] = x[k3];
      }
    }
    float re[4][3], im[4][3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      split<NS>(v[i].x, re[i]);
      split<NS>(v[i].y, im[i]);
    }
    // A: a plane per part and term; B: the two parts of a term are one plane of
    // 2*ROWS rows
    constexpr bool kB = ROWS == TN;
    float* tile = tiles + (int64_t)t * (2 * NS * TILE) + (kB ? kc * (8 * ROWS) + r * 4 : w * 4);
#pragma unroll
    for (int p = 0; p < NS; ++p) {
      *(float4*)(tile + (kB ? 2 * p * TILE : p * TILE)) = make_float4(re[0][p], re[1][p], re[2][p], re[3][p]);
      *(float4*)(tile + (kB ? 2 * p * TILE + 4 * ROWS : (NS + p) * TILE)) =
          make_float4(im[0][p], im[1][p], im[2][p], im[3][p]);
    }
  }
}

// Kahan-compensated sums of two values at a time (sum and compensation as FP32
// pairs; the steps of kahan_add1 on both halves, one instruction each).
struct Kahan2 {
  F2 s, c;
};
__device__ __forceinline__ F2 f2_pack(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void kahan2_add(Kahan2& k, F2 x) {
  const F2 y = f2_sub(x, k.c), t = f2_add(k.s, y);
  k.c = f2_sub(f2_sub(t, k.s), y);
  k.s = t;
}
__device__ __forceinline__ float2 kahan2_value(const Kahan2& k) {
  const float2 s = f2_get(k.s), c = f2_get(k.c);
  return make_float2(s.x - c.x, s.y - c.y);
}

template <int NS>
struct alignas(1024) TcSmem {
  float stage[Cfg<NS>::stages][Cfg<NS>::planes * (kATile + kBTile)];  // A planes, then B planes
  uint64_t full[Cfg<NS>::stages];
  uint64_t empty[Cfg<NS>::stages];
  uint64_t accf[kSets];
  uint64_t acce[kSets];
  uint64_t drain;
  uint32_t tmem_base;
};

// Persistent: each CTA walks output tiles blockIdx.x, +gridDim.x, ... (n tile
// fastest, so the CTAs working on one row block at a time share its A planes
// in L2).  The producer and the MMA issuer run ahead across tile boundaries;
// the epilogue of one tile overlaps the MMAs of the next.
template <typename TC, int NS>
__global__ void __launch_bounds__(kThreads, 1)
    k_tc_gemm(const float* pa, const float* pb, TC* C, const __grid_constant__ GemmDesc d, const int64_t* cm_tab,
              const int64_t* cn_tab, int64_t mtiles, int64_t ntiles, int64_t ktiles, int* status) {
  using CF = Cfg<NS>;
  constexpr int S = CF::stages, P = CF::planes;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  TcSmem<NS>& sm = *reinterpret_cast<TcSmem<NS>*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ntot = ntiles * mtiles * d.Z;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < kSets; ++b) {
      mbar_init(&sm.accf[b], 1);
      mbar_init(&sm.acce[b], kEpiWarps);  // one arrival per epilogue warp
    }
    mbar_init(&sm.drain, 1);
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, kTmemCols);
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = sm.tmem_base;
  bool ok = true;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int64_t g = 0;  // K tiles issued so far (all tiles)
      for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x) {
        const int64_t nt = tile % ntiles, r = tile / ntiles, mt = r % mtiles, z = r / mtiles;
        const float* atile = pa + ((z * mtiles + mt) * ktiles) * (int64_t)(P * kATile);
        const float* btile = pb + ((z * ntiles + nt) * ktiles) * (int64_t)(P * kBTile);
        for (int64_t kt = 0; kt < ktiles; ++kt, ++g) {
          const int s = (int)(g % S);
          const uint32_t ph = (uint32_t)((g / S) & 1);
          if (!mbar_wait(&sm.empty[s], ph ^ 1)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&sm.full[s], CF::stage_bytes);
          float* dst = sm.stage[s];
          bulk_g2s(dst, atile + kt * (P * kATile), P * kATile * 4, &sm.full[s]);
          bulk_g2s(dst + P * kATile, btile + kt * (P * kBTile), P * kBTile * 4, &sm.full[s]);
        }
      }
      // the copies of the last stages are in flight until their full barrier
      // completes: wait (bounded) so none lands after the CTA has exited
      for (int64_t i = g - 1; i >= 0 && i >= g - S; --i)
        if (!mbar_wait(&sm.full[i % S], (uint32_t)((i / S) & 1))) ok = false;
    }
  } else if (warp == 1) {
    // The whole warp runs the loop and waits, one elected thread issues a K
    // tile's MMAs and commits, so that descriptors stay uniform.  Ar.[Br Bi] goes
    // as one N = 128 MMA: 1500 cycles per K tile with two terms, 1650 as N = 64.
    constexpr uint32_t idesc2 = idesc_tf32(TM, 2 * TN), idesc = idesc_tf32(TM, TN),
                       idesc_neg = idesc_tf32(TM, TN, true);
    constexpr uint32_t ALBO = (TM / 8) * 128, BLBO = (2 * TN / 8) * 128, SBO = 128;
    int s = 0, b = 0;  // ring stage and accumulator set, with their phases
    uint32_t ph = 0, use = 0;
    for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x) {
      for (int64_t kt = 0; kt < ktiles; ++kt) {
        if (!__all_sync(0xffffffffu, mbar_wait(&sm.full[s], ph) && mbar_wait(&sm.acce[b], use ^ 1))) {
          ok = false;
          break;
        }
        fence_after();
        const uint32_t sa = smem_u32(sm.stage[s]) >> 4;
        const uint32_t sb = sa + ((P * kATile * 4) >> 4);
        const uint32_t dr = tmem + (uint32_t)b * (2 * TN), di = dr + TN;
        // The tensor core rounds an accumulation toward zero.  The small
        // correction products go in first (the first one overwrites), the
        // large hi x hi products last.
        if (elect_one()) {
#pragma unroll
          for (int q = 1; q <= CF::products; ++q) {
            const int qq = q == CF::products ? 0 : q;  // hi x hi last
            // term pairs (i, j) with i + j < NS: (0,0) (0,1) (1,0) (0,2) (2,0) (1,1)
            const int ti = (qq == 2) ? 1 : (qq == 4) ? 2 : (qq == 5) ? 1 : 0;
            const int tj = (qq == 1) ? 1 : (qq == 3) ? 2 : (qq == 5) ? 1 : 0;
#pragma unroll
            for (int j = 0; j < TK / 8; ++j) {  // the two 8-deep halves of the tile
              const uint32_t acc = (q == 1 && j == 0) ? 0u : 1u;
              const uint32_t oa = (uint32_t)j * 2 * ALBO, ob = (uint32_t)j * 2 * BLBO;
              const uint64_t ar = desc_at(sa + (((0 * NS + ti) * kATile * 4 + oa) >> 4), ALBO, SBO);
              const uint64_t ai = desc_at(sa + (((1 * NS + ti) * kATile * 4 + oa) >> 4), ALBO, SBO);
              const uint64_t br = desc_at(sb + ((tj * 2 * kBTile * 4 + ob) >> 4), BLBO, SBO);
              const uint64_t bi = desc_at(sb + ((tj * 2 * kBTile * 4 + ob + TN * 16) >> 4), BLBO, SBO);
              mma_tf32(dr, ar, br, idesc2, acc);    // + Ar.[Br Bi]
              mma_tf32(dr, ai, bi, idesc_neg, 1u);  // - Ai.Bi
              mma_tf32(di, ai, br, idesc, 1u);      // + Ai.Br
            }
          }
          mma_commit(&sm.accf[b]);   // chunk accumulators ready for the epilogue
          mma_commit(&sm.empty[s]);  // smem stage free once these MMAs finish
        }
        if (++s == S) {
          s = 0;
          ph ^= 1u;
        }
        if (++b == kSets) {
          b = 0;
          use ^= 1u;
        }
      }
    }
    // every MMA issued has finished once this arrives (TMEM is freed below)
    if (elect_one()) mma_commit(&sm.drain);
    if (!mbar_wait(&sm.drain, 0)) ok = false;
  } else {
    // epilogue: warp w reads TMEM lanes of quadrant w % 4, columns [16h, 16h+16)
    constexpr int CW = TN / (kEpiWarps / 4);  // columns per epilogue warp
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    int b = 0;
    uint32_t use = 0;
    for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x) {
      const int64_t nt = tile % ntiles, r = tile / ntiles, mt = r % mtiles, z = r / mtiles;
      const int64_t m = mt * TM + row, n0 = nt * TN + h * CW;
      const int ncol = (int)(d.N - n0 < CW ? d.N - n0 : CW);  // columns of this warp inside C (may be <= 0)
      // result offsets, loaded ahead of the sums: this lane's row (-1: outside C)
      // and the column n0 + lane
      const int64_t base = m < d.M ? decode(z, d.nz, d.zdim, d.zsc) + cm_tab[m] : -1;
      const int64_t coff = lane < ncol ? cn_tab[n0 + lane] : 0;
      Kahan2 ar[CW / 2], ai[CW / 2];  // sums of the real and imaginary parts, two columns each
#pragma unroll
      for (int j = 0; j < CW / 2; ++j) ar[j] = ai[j] = Kahan2{0, 0};
      for (int kt = (int)ktiles; kt > 0; --kt) {
        // the TMEM loads below are warp-collective
        if (!__all_sync(0xffffffffu, mbar_wait(&sm.accf[b], use))) {
          ok = false;
          break;
        }
        fence_after();
        const uint32_t col = (uint32_t)(b * 2 * TN + h * CW);
        // eight columns at a time: 64 registers of sums and 16 of values fit the
        // 112 that 18 warps leave a thread
#pragma unroll
        for (int c = 0; c < CW; c += 8) {
          float vr[8], vi[8];
          tmem_ld8(lane_base + col + c, vr);
          tmem_ld8(lane_base + col + c + TN, vi);
          tmem_wait_ld();
          if (c + 8 == CW) {  // values are in registers: hand the set back
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.acce[b]);
          }
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            kahan2_add(ar[(c + j) / 2], f2_pack(vr[j], vr[j + 1]));
            kahan2_add(ai[(c + j) / 2], f2_pack(vi[j], vi[j + 1]));
          }
        }
        if (++b == kSets) {
          b = 0;
          use ^= 1u;
        }
      }
      if (!ok) break;
      // lane j holds the result offset of column n0 + j: adjacent columns leave as
      // 32-byte stores where they are adjacent (and aligned) in C too
      const int64_t cn_prev = __shfl_up_sync(0xffffffffu, coff, 1);
      const uint32_t step = __ballot_sync(0xffffffffu, lane < ncol && coff == cn_prev + 1);
#pragma unroll
      for (int c = 0; c < CW; c += 4) {
        float2 v[4];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          // the truncations of every chunk shrink it by kTruncBias relative
          // on average; the sum is linear in the chunks, so the expectation
          // is added back once here
          const float2 re = kahan2_value(ar[(c + j) / 2]), im = kahan2_value(ai[(c + j) / 2]);
          v[j] = make_float2(fmaf(kTruncBias, re.x, re.x), fmaf(kTruncBias, im.x, im.x));
          v[j + 1] = make_float2(fmaf(kTruncBias, re.y, re.y), fmaf(kTruncBias, im.y, im.y));
        }
        int64_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = base + __shfl_sync(0xffffffffu, coff, c + j);
        if (base < 0) continue;
        if constexpr (sizeof(TC) == 8) {
          if (((step >> (c + 1)) & 7u) == 7u && ((uintptr_t)(C + o[0]) & 31) == 0) {
            asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(C + o[0]), "f"(v[0].x), "f"(v[0].y),
                         "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y)
                         : "memory");
            continue;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < ncol) C[o[j]] = store_as<TC>(v[j]);
      }
    }
  }
  if (!ok) report_timeout(status);
  fence_before();
  __syncthreads();
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

int splits_of(int precision) { return precision == PQ_PREC_6XTF32 ? 3 : 2; }

template <typename T, int NS, int ROWS>
cudaError_t pack(const void* X, float* planes, const GemmDesc& d, int side, int64_t rows, int64_t rtiles, int64_t kt,
                 cudaStream_t s) {
  // as many K tiles per block as leave the SMs four blocks each
  const int64_t kper = std::max<int64_t>(1, std::min<int64_t>(kPackMaxK, kt * rtiles * d.Z / (4 * sm_count())));
  const dim3 grid((unsigned)ceil_div(kt, kper), (unsigned)rtiles, (unsigned)d.Z);
  return launch_pdl(k_tc_pack<T, NS, ROWS>, grid, dim3(256), 0, s, (const T*)X, planes, d, side, rows, rtiles, kt,
                    (int)kper);
}
template <int NS>
cudaError_t pack_both(const void* A, int ta, const void* B, int tb, float* pa, float* pb, const GemmDesc& d,
                      int64_t mt, int64_t nt, int64_t kt, cudaStream_t s) {
  cudaError_t e = ta == PQ_C128 ? pack<double2, NS, TM>(A, pa, d, 0, d.M, mt, kt, s)
                                : pack<float2, NS, TM>(A, pa, d, 0, d.M, mt, kt, s);
  if (e != cudaSuccess) return e;
  return tb == PQ_C128 ? pack<double2, NS, TN>(B, pb, d, 1, d.N, nt, kt, s)
                       : pack<float2, NS, TN>(B, pb, d, 1, d.N, nt, kt, s);
}

template <typename TC, int NS>
cudaError_t gemm_launch(const float* pa, const float* pb, void* C, const GemmDesc& d, const int64_t* cm,
                        const int64_t* cn, int64_t mt, int64_t nt, int64_t kt, int* status, cudaStream_t s) {
  static_assert(sizeof(TcSmem<NS>) + 1024 <= 232448, "shared memory layout exceeds 227 KiB");
  // the whole opt-in shared memory (one CTA per SM either way): the ring plus
  // slack past the last stage
  const size_t smem = 232448;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k_tc_gemm<TC, NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int64_t tiles = mt * nt * d.Z;
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, sm_count());
  return launch_pdl(k_tc_gemm<TC, NS>, dim3(grid), dim3(kThreads), smem, s, pa, pb, (TC*)C, d, cm, cn, mt, nt, kt,
                    status);
}

}  // namespace

// PQ_PREC_OZAKI / PQ_PREC_OZAKI4 / PQ_PREC_3XBF16 run the exact-accumulation
// kernels (pq_oz.cu: 5 / 4 / 3 bf16 slices, for the first with complex64 results
// and K <= 256 four fp16 ones) where their limits allow (K <= 512) and the
// 6xTF32 (the first two) / 3xTF32 kernels otherwise.
static bool tf32_eligible(const GemmDesc& d) {
  if (d.M < 64 || d.N < 64 || d.K < 16) return false;
  return d.Z <= 65535 && ceil_div(d.N, TN) <= 65535 && ceil_div(d.M, TM) <= 65535;
}
static int tf32_precision(int precision) {
  return (precision == PQ_PREC_OZAKI || precision == PQ_PREC_OZAKI4)
             ? PQ_PREC_6XTF32
             : (precision == PQ_PREC_3XBF16 ? PQ_PREC_3XTF32 : precision);
}
static bool sliced(int precision) {
  return precision == PQ_PREC_OZAKI || precision == PQ_PREC_OZAKI4 || precision == PQ_PREC_3XBF16;
}
// The bf16 slices of the mode (its scratch is sized for them: planes of four
// fp16 slices take less).
static int mode_slices(int precision) {
  return precision == PQ_PREC_OZAKI ? 5 : (precision == PQ_PREC_OZAKI4 ? 4 : 3);
}

size_t tc_scratch_bytes(int precision, const GemmDesc& d) {
  if (sliced(precision) && oz_eligible(d)) return oz_scratch_bytes(mode_slices(precision), d);
  const int P = 2 * splits_of(tf32_precision(precision));
  const int64_t mt = ceil_div(d.M, TM), nt = ceil_div(d.N, TN), kt = ceil_div(d.K, TK);
  return (size_t)(d.Z * (mt * kATile + nt * kBTile) * kt * P * 4) + (size_t)(d.M + d.N) * 8 + 1024;
}

bool tc_eligible(int precision, const GemmDesc& d) {
  if (precision != PQ_PREC_3XTF32 && precision != PQ_PREC_6XTF32 && !sliced(precision)) return false;
  if (sliced(precision) && oz_eligible(d)) return true;
  return tf32_eligible(d) && tc_scratch_bytes(precision, d) <= (size_t(24) << 30);
}

int tc_launch_count(int precision, const GemmDesc& d) {
  // exponents of A and B, slices of B, result index table, GEMM (A is sliced
  // inside it); or the TF32 path's index table, two packs, GEMM
  return (sliced(precision) && oz_eligible(d)) ? 5 : 4;
}

cudaError_t launch_tc(int precision, int ta, int tb, int tc, const void* A, const void* B, void* C, const GemmDesc& d,
                      void* scratch, size_t scratch_bytes, int* status, cudaStream_t stream) {
  if (!tc_eligible(precision, d)) return cudaErrorNotSupported;
  if (!scratch || scratch_bytes < tc_scratch_bytes(precision, d)) return cudaErrorInvalidValue;
  if (sliced(precision) && oz_eligible(d))
    return launch_oz(mode_slices(precision), ta, tb, tc, A, B, C, d, scratch, scratch_bytes, status, stream);
  const int NS = splits_of(tf32_precision(precision));
  const int64_t mt = ceil_div(d.M, TM), nt = ceil_div(d.N, TN), kt = ceil_div(d.K, TK);
  float* pa = (float*)(((uintptr_t)scratch + 255) & ~(uintptr_t)255);
  float* pb = pa + d.Z * mt * kt * (int64_t)(2 * NS * kATile);
  int64_t* cm = (int64_t*)(pb + d.Z * nt * kt * (int64_t)(2 * NS * kBTile));
  int64_t* cn = cm + d.M;
  const int64_t idx_blocks = std::min<int64_t>(ceil_div(d.M + d.N, 256), 152 * 8);
  cudaError_t e = launch_pdl(k_result_index<0>, dim3((unsigned)idx_blocks), dim3(256), 0, stream, d, cm, cn);
  if (e != cudaSuccess) return e;
  if (NS == 2) {
    if ((e = pack_both<2>(A, ta, B, tb, pa, pb, d, mt, nt, kt, stream)) != cudaSuccess) return e;
    return tc == PQ_C128 ? gemm_launch<double2, 2>(pa, pb, C, d, cm, cn, mt, nt, kt, status, stream)
                         : gemm_launch<float2, 2>(pa, pb, C, d, cm, cn, mt, nt, kt, status, stream);
  }
  if ((e = pack_both<3>(A, ta, B, tb, pa, pb, d, mt, nt, kt, stream)) != cudaSuccess) return e;
  return tc == PQ_C128 ? gemm_launch<double2, 3>(pa, pb, C, d, cm, cn, mt, nt, kt, status, stream)
                       : gemm_launch<float2, 3>(pa, pb, C, d, cm, cn, mt, nt, kt, status, stream);
}

}  // namespace pq
