// Exact-accumulation split-precision complex contraction on the tcgen05 tensor
// cores (sm_103a, PQ_PREC_OZAKI): the Ozaki scheme (Ozaki, Ogita, Oishi, Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applicability", Numer. Algorithms 59, 2012)
// with 16-bit slices and FP32 accumulation in TMEM.
//
// Scaling.  Every row m of A (over K, per batch index) gets the power of two
// 2^ea[m] with every |Re|, |Im| of the row below it (frexp exponent of the row
// maximum); likewise every column n of B gets 2^eb[n].  A scaled value
// x = a 2^-ea in (-1, 1) is cut into slices, and the products of A's slice i
// and B's slice j are accumulated by level i + j into three FP32 accumulators
// per real output (Cr, Ci): level 0, level 1 and the rest.
//
// Five bf16 slices (PQ_PREC_OZAKI: complex128 results, and complex64 ones with
// K > 256)
//   s0 = rint(x 2^7) 2^-7,  s_i = rint((x - s0 - .. - s_{i-1}) 2^{7(i+1)}) 2^{-7(i+1)}
// (|s0| <= 1, |s_i| <= 2^{-7i-1}), each an integer of at most 8 bits times a
// power of two, hence exact in bf16; x - (s0 + .. + s4) is below 2^-36, so a
// value 2^-10 below its row maximum still keeps 26 significant bits.  s_i t_j is
// an integer multiple of 2^{-7(i+j+2)} of magnitude at most 2^{-7(i+j)}; the 15
// slice pairs with i + j <= 4 are accumulated:
//   level 0   (0,0)             multiples of 2^-14, |sum| <= 2K
//   level 1   (0,1) (1,0)       multiples of 2^-21, |sum| <= 4K 2^-8
//   levels 2-4 (the other 12)   |sum| <= 2^-14 relative
// For K <= 512 the level-0 and level-1 sums are exact in FP32; only the small
// levels 2-4 round (toward zero, K / 16 times per pair).  The result is
// (L0 + L1 + L2) 2^(ea+eb) rounded once to the output type, so the error is
// the output rounding, the dropped pairs and slice residuals, at most 2^-33 K
// 2^(ea+eb) per component, and the rest's roundings (rms 2^-34 of the scales
// for K = 16, 2^-30 for 256, 2^-28 for 512 on random operands).  (Four 7-bit
// slices, ten pairs, double the amplitude error of deep circuits: their rows
// span many binades.)
//
// Four fp16 slices (kHalf, PQ_PREC_OZAKI with complex64 results and K <= 256): s0
// on a grid of 2^-8 or 2^-7, s1 on one 8 or 7 bits finer (first_bits,
// second_bits: as fine as leaves levels 0 and 1 exact in FP32 whatever the
// operands are), s2 the remainder in fp16's 11 bits, s3 the rest of that, so
// x - (s0 + .. + s3) is at most 2^-39.  11 pairs: all but (1,3) (3,1) (2,3)
// (3,2) (3,3), at most 2^-35 in all, where the five bf16 slices drop 2^-35 and
// have twice a residual of 2^-36.  The rest takes 8 pairs of the same sizes
// instead of 12.  So no operand keeps fewer bits and no error is larger than
// with the five slices, and 11 products do (rest's rms 2^-36 for K = 16, 2^-30.2
// for 256).  Three fp16 slices with 12 bits in s1 (8 products) were faster and not
// sound: level 1 then has up to 29 bits for the accumulator's 24, which shows
// where level 0 cancels (K = 512, A alternating +-0.75 plus 2^-8: error 1.3e-6 of
// the scales, 3e-8 with level 1 exact).
//   Cr = Ar.Br + (-Ai).Bi   (the negation is the MMA's negate-A bit)
//   Ci = Ar.Bi + Ai.Br
//
// Complex arithmetic on real tensor cores: a tile of 64 complex rows of A is
// held as the 192-row stack [Ar; Ai; -Ar] of each slice, so that
//   X1 = rows 0..127   = [Ar; Ai]
//   X2 = rows 64..191  = [Ai; -Ar]  (issued with the MMA's negate-A bit: [-Ai; Ar])
// and one accumulator of 128 TMEM lanes receives
//   X1 . Br + X2' . Bi = [Ar.Br - Ai.Bi ; Ai.Br + Ar.Bi] = [Cr ; Ci]
// for the 64 rows: 2 MMAs (M=128, N=TN, K=16) per slice pair and K tile.
//
// Kernels (one launch each, in stream order):
//   k_oz_exp        row scale exponents of A (k_oz_exp_k when A is contiguous
//                   along K), column scale exponents of B
//   k_oz_pack       B's slices into planes [z][col tile][k tile][plane][TN*16
//                   16-bit values] in the canonical no-swizzle K-major layout
//                   (8-row x 16-byte core matrices), planes {Re s0.., Im
//                   s0..}; columns and K beyond the operand are 0
//   k_result_index  result offsets of every row and column of C
//   k_oz_gemm       persistent, one CTA per SM over 64 x TN complex output
//                   tiles (TN = 128, or 64 / 32 / 16 for narrow pairs; a pair
//                   whose A side is the narrow one runs as B x A):
//     warp 0       producer: cp.async.bulk of B's plane tiles of one
//                  16-deep K tile into B's shared-memory ring;
//     warp 1       TMEM owner and MMA issuer: 22 tcgen05.mma (kind::f16; 30
//                  for five slices) per K tile into three TN-column
//                  accumulators (levels 0, 1, rest); narrow tiles (TN <= 64)
//                  alternate between two such sets, so a tile's MMAs do not
//                  wait for the epilogue of the one before; 16-wide tiles
//                  issue one MMA per A slice i against the B slices it meets
//                  side by side, each slice pair into its own 16-column
//                  region;
//     8 or 12 warps A converters: gather A's 64 x 16 complex values of the K
//                  tile through its index map straight from HBM (the group's
//                  next K tile in flight while this one is sliced), slice
//                  them and store the [Ar; Ai; -Ar] stacks into A's ring (no
//                  slice planes of A ever reach HBM); for complex64 A two
//                  or three groups of four warps take K tiles in turn, each
//                  thread 8 consecutive k of one row, so every store is a
//                  whole 16-byte core-matrix row;
//     8 or 4 warps  epilogue, once per tile: Cr from TMEM lanes 0-63, Ci from
//                  lanes 64-127; the levels are combined with an error-free
//                  two-sum (128-wide complex64 tiles park the sums, in shared
//                  memory or the spare TMEM block, and release the
//                  accumulators first), scaled by 2^(ea+eb) and scattered
//                  through the result index map.
// Every mbarrier wait is bounded; on expiry the kernel records an error in the
// context's status word and runs to the end (TMEM is always released).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "pq_tcgen05.cuh"
#include "pq_types.cuh"

namespace pq {

namespace {

using namespace tcg;

constexpr int TK = 16;
constexpr int kThreads = 576;                    // producer, MMA, 16 converter and epilogue warps
constexpr int kWorkWarps = 16;                   // converter + epilogue warps
constexpr int kRows = 64;                        // complex rows of A per tile
constexpr int kStackBytes = 3 * kRows * TK * 2;  // one slice's [Ar; Ai; -Ar] stack (6 KiB)
constexpr int kExpZero = -4096;                  // exponent of an all-zero row
constexpr int64_t kMaxK = 512;                   // exact level-0/1 sums up to this K

// Tile width N: 128 for general pairs, 64 / 32 / 16 for narrow ones.
// Split of a real value: kHalf for PQ_PREC_OZAKI with complex64 results and K <=
// kHalfMaxK (four fp16 slices, 11 pairs); bf16 slices for the others: 5 for
// PQ_PREC_OZAKI (15 slice pairs, i + j <= 4), 4 for PQ_PREC_OZAKI4 (10 pairs,
// i + j <= 3), 3 for PQ_PREC_3XBF16 (6 pairs, i + j <= 2).
constexpr int kHalf = 8;
constexpr int64_t kHalfMaxK = 256;
template <int S>
struct Sl {
  static_assert(S == kHalf || S == 5 || S == 4 || S == 3, "split");
  static constexpr bool half = S == kHalf;
  static constexpr int n = half ? 4 : S;      // slices
  static constexpr int planes = 2 * n;        // per operand: Re s0.., Im s0..
  static constexpr int pairs = half ? 11 : (S == 5 ? 15 : (S == 4 ? 10 : 6));
  // slices 0 .. met(i) - 1 of B meet slice i of A
  __host__ __device__ static constexpr int met(int i) {
    return half ? (i == 0 ? 4 : (i == 3 ? 1 : 3)) : n - i;
  }
};
// Converter warps (the rest are epilogue warps): 8; 12 for 16-wide tiles of more
// than six K tiles of complex64 A in fp16 slices, whose few MMAs wait for A's
// loads -- a third group of converters keeps half as much again in flight
// (2^18 rows, N = 16, K = 256: 337 -> 306 us; a second K tile per thread
// spilled).  Shorter tiles wait for their stores (K = 64: 142 us with 12, 125
// with 8), 32-wide ones for their MMAs (K = 48: 180 and 134 us, K = 256: 357 and
// 354).
template <typename TA, int TN, int S>
__host__ __device__ constexpr bool many_converters() {
  return TN == 16 && Sl<S>::half && sizeof(TA) == 8;
}
// kHalf: scaled values are held times 2^kHalfUp, so that the lowest bits of
// the last slice stay in fp16's range (its subnormals, 2^-24, are 2^-39).
constexpr int kHalfUp = 15;
// Bits of the first slice (a grid of 2^-bits) and how many more the second has.
// With a and b first bits and K terms of two real products, a level-0 sum is at
// most 2K on a grid of 2^-(a+b): 24 bits for a + b + 1 + log2 K <= 24, so 8 and 8
// for K <= 128, 7 and 8 for K <= 256.  Level 1 is at most 2K (2^-(a+1) + 2^-(b+1))
// on a grid of 2^-(a+b+more): 1 and 2^-24 for K <= 128 with 8 more bits, 3 and
// 2^-22 for K <= 256 with 7 more.
__host__ __device__ constexpr int first_bits(int64_t k, int side) { return k <= (side == 0 ? 128 : 256) ? 8 : 7; }
__host__ __device__ constexpr int second_bits(int64_t k) { return k <= 128 ? 8 : 7; }

// 128-wide tiles of kHalf or three slices with complex64 results: the epilogue
// parks a tile's sums in shared memory (and stores whole complex values from
// there), and the fourth TMEM block lets the next tile's MMAs of levels 2 and up
// start before the epilogue has read this one.  Against parking in the fourth
// block with a ring of three stages (kHalf): 2^20 x 256 x 16 in 1.44 instead of
// 2.36 ms, 2^18 x 128 x 64 in 0.27 instead of 0.39; K = 256, where two stages of
// A are the price, 4.26 instead of 4.17.
template <typename TC, int TN, int S>
__host__ __device__ constexpr bool oz_park() {
  return TN == 128 && (Sl<S>::half || S == 3) && sizeof(TC) == 8;
}

template <int TN, int S, bool PARK>
struct OzCfg {
  static constexpr int kBTile = TN * TK;                                   // 16-bit values per B plane tile
  static constexpr uint32_t b_bytes = Sl<S>::planes * kBTile * 2;          // B planes of one K tile
  static constexpr uint32_t a_bytes = Sl<S>::n * kStackBytes;              // A stacks of one K tile
  // Rings of A stacks and of B planes.  Beside parked sums 227 KB hold two
  // stages of four slices of A (24 KB) and three of B (32 KB): A's stores are
  // short once a stage is free, B's copies take their time.
  static constexpr int b_stages = PARK ? 3 : (Sl<S>::half ? (TN == 64 ? 5 : 6) : ((TN == 128 && S >= 4) ? 3 : 4));
  static constexpr int a_stages = PARK && Sl<S>::half ? 2 : b_stages;
  // rings of one length are one ring: a stage of both has one pair of barriers
  static constexpr bool one_ring = a_stages == b_stages;
  // 16-wide tiles: one MMA per A slice i against B slices 0 .. met(i)-1 side
  // by side (N = 16 met(i)), every slice pair in its own TMEM region
  static constexpr bool narrow = TN == 16;
  // accumulator columns of one tile: three levels of TN columns, or the pair
  // regions of 16 columns
  static constexpr int set_cols = narrow ? 16 * Sl<S>::pairs : 3 * TN;
  // accumulator sets: two for TN <= 64, so that the MMAs of the next tile
  // run while the epilogue drains this one
  static constexpr int acc_sets = TN <= 64 ? 2 : 1;
  static constexpr uint32_t tmem_cols =
      TN == 128 ? 512 : (TN == 64 ? 512 : (TN == 32 ? 256 : (2 * set_cols > 256 ? 512 : 256)));
  static_assert(acc_sets * set_cols <= (int)tmem_cols && a_bytes % 1024 == 0 && b_bytes % 1024 == 0, "tile width");
};

// First TMEM column of A slice i's region in a narrow tile.
template <int S>
__host__ __device__ constexpr int narrow_col(int i) {
  int c = 0;
  for (int q = 0; q < i; ++q) c += 16 * Sl<S>::met(q);
  return c;
}

// Slice pairs, level 0 first, then level 1, then the rest with the smallest
// first.  The order in which the bf16 splits issue them (the truncating rest
// accumulator then takes the fewest additions at full size: by slice of A from
// the first its rms error is 5 to 17 % larger, K = 512 to 64), and in which the
// epilogue of 16-wide tiles adds the pairs' regions up.  Five slices:
//   i: 0 0 1 0 1 2 3 4 0 1 2 3 0 1 2
//   j: 0 1 0 4 3 2 1 0 3 2 1 0 2 1 0
// four slices (levels 0 to 3, ten pairs):
//   i: 0 0 1 0 1 2 3 0 1 2
//   j: 0 1 0 3 2 1 0 2 1 0
// three slices:
//   i: 0 0 1 0 1 2
//   j: 0 1 0 2 1 0
// kHalf:
//   i: 0 0 1 2 3 0 2 1 2 0 1
//   j: 0 1 0 2 0 3 1 2 0 2 1
// (4-bit fields, pair p in bits [4p, 4p + 4))
template <int S>
__host__ __device__ constexpr int pair_i(int p) {
  return (int)((S == kHalf ? 0x10212032100ull
                           : (S == 5 ? 0x210321043210100ull : (S == 4 ? 0x2103210100ull : 0x210100ull))) >>
               (4 * p)) &
         15;
}
template <int S>
__host__ __device__ constexpr int pair_j(int p) {
  return (int)((S == kHalf ? 0x12021302010ull
                           : (S == 5 ? 0x12012301234010ull : (S == 4 ? 0x0120123010ull : 0x12010ull))) >>
               (4 * p)) &
         15;
}

template <typename T>
struct Real;
template <>
struct Real<float2> {
  using R = float;
};
template <>
struct Real<double2> {
  using R = double;
};

__device__ __forceinline__ float absmax(float a, float b) { return fmaxf(fabsf(a), fabsf(b)); }
__device__ __forceinline__ double absmax(double a, double b) { return fmax(fabs(a), fabs(b)); }
__device__ __forceinline__ float scale2(float x, int e) { return ldexpf(x, e); }
__device__ __forceinline__ double scale2(double x, int e) { return ldexp(x, e); }
__device__ __forceinline__ float round_int(float x) { return rintf(x); }
__device__ __forceinline__ double round_int(double x) { return rint(x); }

__device__ __forceinline__ int exp_of(float v) {
  int e;
  frexpf(v, &e);
  return v == 0.f ? kExpZero : e;
}
__device__ __forceinline__ int exp_of(double v) {
  int e;
  frexp(v, &e);
  return v == 0.0 ? kExpZero : e;
}

// Row (side 0: A rows m) or column (side 1: B columns n) scale exponents:
// e[z * rows + r] = frexp exponent of the largest |Re|, |Im| over k.
// One block per (ROWS-row tile, z); thread t always reads row t % ROWS (K
// offsets staged in shared memory), keeps a running maximum with four loads
// in flight, and the 256 / ROWS threads of a row combine at the end.
template <typename T, int ROWS>
__global__ void __launch_bounds__(256) k_oz_exp(const T* __restrict__ X, const __grid_constant__ GemmDesc d, int side,
                                                int64_t rows, int* __restrict__ e_out) {
  static_assert(256 % ROWS == 0, "rows per block");
  constexpr int KS = 256 / ROWS;  // threads per row
  __shared__ int64_t koff[kMaxK];
  __shared__ int emax[ROWS];
  const int64_t rt = blockIdx.x, z = blockIdx.y;
  const int nrm = side == 0 ? d.nm : d.nn;
  const int64_t* rdim = side == 0 ? d.mdim : d.ndim;
  const int64_t* rstr = side == 0 ? d.msa : d.nsb;
  const int64_t* kstr = side == 0 ? d.ksa : d.ksb;
  const int64_t* zstr = side == 0 ? d.zsa : d.zsb;
  for (int t = threadIdx.x; t < ROWS; t += blockDim.x) emax[t] = kExpZero;
  for (int t = threadIdx.x; t < d.K; t += blockDim.x) koff[t] = decode32(t, d.nk, d.kdim, kstr);
  __syncthreads();
  using R = typename Real<T>::R;
  const int r = threadIdx.x % ROWS, k0 = threadIdx.x / ROWS;
  const int64_t row = rt * ROWS + r;
  if (row < rows) {
    const T* xr = X + decode32(z, d.nz, d.zdim, zstr) + decode32(row, nrm, rdim, rstr);
    R mx = 0;
    int64_t k = k0;
    for (; k + 3 * KS < d.K; k += 4 * KS) {
      const T v0 = xr[koff[k]], v1 = xr[koff[k + KS]], v2 = xr[koff[k + 2 * KS]], v3 = xr[koff[k + 3 * KS]];
      mx = fmax(mx, fmax(fmax(absmax((R)v0.x, (R)v0.y), absmax((R)v1.x, (R)v1.y)),
                         fmax(absmax((R)v2.x, (R)v2.y), absmax((R)v3.x, (R)v3.y))));
    }
    for (; k < d.K; k += KS) {
      const T v = xr[koff[k]];
      mx = fmax(mx, absmax((R)v.x, (R)v.y));
    }
    atomicMax(&emax[r], exp_of(mx));
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ROWS; t += blockDim.x) {
    const int64_t rr = rt * ROWS + t;
    if (rr < rows) e_out[z * rows + rr] = emax[t];
  }
}

// Four complex64 values (32 bytes, 32-byte aligned) of a read-only operand.
__device__ __forceinline__ void ldg256(const void* p, float* v) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(p));
}

// Row scale exponents of A when A is contiguous along K (its first K mode has
// stride 1 and extent >= 2) but not along M: KL consecutive lanes read the
// values of one row, V adjacent ones each (V = 4: complex64 that k_vector
// allows, one 32-byte load), combine their maxima with shuffles, and the
// RS = 32 / KL row groups of a warp take consecutive rows.  V * KL is at most A's
// leading contiguous run of K (all K modes that continue it in A, in
// whatever order B has them), so that a load of a warp covers whole runs.  A
// warp takes four rows per lane group (no branch between their loads, so that
// eight are in flight per lane), a block 8 warps; one z per blockIdx.y.
// Bound by reading A once: 2^20 rows of 256 complex64 in runs of 16 take
// 323 us, 6.6 TB/s (537 us when only K modes merged with B's counted as a run:
// two values per row and load).
template <typename T, int V>
__global__ void __launch_bounds__(256) k_oz_exp_k(const T* __restrict__ X, const __grid_constant__ GemmDesc d,
                                                  int64_t rows, int KL, int* __restrict__ e_out) {
  using R = typename Real<T>::R;
  __shared__ int64_t koff[kMaxK];
  const int64_t z = blockIdx.y;
  for (int t = threadIdx.x; t < d.K; t += blockDim.x) koff[t] = decode32(t, d.nk, d.kdim, d.ksa);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int RS = 32 / KL;
  const int sub = lane / KL, kl = lane % KL;
  const int64_t zo = decode32(z, d.nz, d.zdim, d.zsa);
  const int64_t r0 = ((int64_t)blockIdx.x * 8 + warp) * 4 * RS + sub;
  const T* xr[4];
  R mx[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // rows past the end read the last row (and store nothing)
    const int64_t row = r0 + i * RS < rows ? r0 + i * RS : rows - 1;
    xr[i] = X + zo + decode32(row, d.nm, d.mdim, d.msa);
    mx[i] = 0;
  }
#pragma unroll 2
  for (int k = V * kl; k < d.K; k += V * KL) {
    const int64_t o = koff[k];
    if constexpr (V == 4) {
      float f[4][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) ldg256(xr[i] + o, f[i]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 8; q += 2) mx[i] = fmaxf(mx[i], absmax(f[i][q], f[i][q + 1]));
    } else {
      T y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = xr[i][o];
#pragma unroll
      for (int i = 0; i < 4; ++i) mx[i] = fmax(mx[i], absmax((R)y[i].x, (R)y[i].y));
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    for (int s = KL / 2; s > 0; s >>= 1) mx[i] = fmax(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], s));
    if (kl == 0 && r0 + i * RS < rows) e_out[z * rows + r0 + i * RS] = exp_of(mx[i]);
  }
}

// Whether the exponent pass and the converters may read complex64 A as aligned
// 32-byte runs of four K values: the leading K modes that follow each other in A
// (in whatever order B has them) make a run from stride 1 whose extent is a
// multiple of 4 (so runs of 4 from a multiple of 4 never cross it), and every
// other stride and the base keep the alignment.  Otherwise they read value by
// value, which coalesces over rows when A's first M mode has stride 1; over rows
// 128 bytes apart it costs the converters a wavefront of the L1 per row and
// value, 88 % of its rate (2^20 x 256 x 256 with runs of 16, exponent pass
// included: 3.35 ms value by value, 2.75 so, with 8 products per pair).
bool k_vector(const void* A, const GemmDesc& d) {
  if (((uintptr_t)A & 31) || d.nk < 1 || d.ksa[0] != 1) return false;
  int64_t run = d.kdim[0];
  int lead = 1;
  for (; run % 4 && lead < d.nk && d.ksa[lead] == run; ++lead) run *= d.kdim[lead];
  if (run % 4) return false;
  for (int i = lead; i < d.nk; ++i)
    if (d.ksa[i] % 4) return false;
  for (int i = 0; i < d.nm; ++i)
    if (d.msa[i] % 4) return false;
  for (int i = 0; i < d.nz; ++i)
    if (d.zsa[i] % 4) return false;
  return true;
}

// A's row exponents: the K-major kernel when A's first K mode has stride 1
// (and its first M mode does not), else the row-per-thread kernel.
template <typename T>
void row_exponents(const T* A, const GemmDesc& d, int* ea, cudaStream_t s) {
  if (d.nk > 0 && d.ksa[0] == 1 && d.kdim[0] >= 2 && !(d.nm > 0 && d.msa[0] == 1)) {
    int64_t run = d.kdim[0];  // K values adjacent in A
    for (int i = 1; i < d.nk && d.ksa[i] == run; ++i) run *= d.kdim[i];
    const bool four = sizeof(T) == 8 && k_vector(A, d);
    int KL = 1;
    while (KL < 32 && 2 * KL * (four ? 4 : 1) <= run) KL *= 2;
    const dim3 grid((unsigned)ceil_div(d.M, 8 * 4 * (32 / KL)), (unsigned)d.Z);
    if constexpr (sizeof(T) == 8)
      if (four) {
        k_oz_exp_k<T, 4><<<grid, 256, 0, s>>>(A, d, d.M, KL, ea);
        return;
      }
    k_oz_exp_k<T, 1><<<grid, 256, 0, s>>>(A, d, d.M, KL, ea);
  } else {
    k_oz_exp<T, 128><<<dim3((unsigned)ceil_div(d.M, 128), (unsigned)d.Z), 256, 0, s>>>(A, d, 0, d.M, ea);
  }
}

// The bf16 slices of x (|x| < 1 after scaling); every step is exact in R.
template <typename R, int NSL>
__device__ __forceinline__ void slices(R x, float* s) {
  R r = x;
  R g = (R)128.0, gi = (R)(1.0 / 128.0);  // 2^7(i+1) and its inverse (exact)
#pragma unroll
  for (int i = 0; i < NSL; ++i) {
    const R si = round_int(r * g) * gi;
    s[i] = (float)si;
    r -= si;
    g *= (R)128.0;
    gi *= (R)(1.0 / 128.0);
  }
}
// x rounded to a multiple of 2^e for |x| < 2^(e + 21), by adding and taking
// off c = 1.5 2^(23 + e).
__device__ __forceinline__ float round_grid(float x, float c) { return __fadd_rn(__fadd_rn(x, c), -c); }
// v rounded to fp16's 11 bits.
__device__ __forceinline__ float round_half(float v) { return __half2float(__float2half_rn(v)); }
// The fp16 slices of x 2^kHalfUp (|x| < 1): s0 on the grid of c0, s1 on the
// grid of c1, s2 the remainder rounded to 11 bits, s3 the rest of that (rounded to
// 11 bits, or multiples of 2^-24, when it is stored).  Exact but for that last
// rounding; |s1| and |s2| are at most half a step of the slice before.
__device__ __forceinline__ void half_slices(float x, float c0, float c1, float* s) {
  s[0] = round_grid(x, c0);
  float r = x - s[0];
  s[1] = round_grid(r, c1);
  r -= s[1];
  s[2] = round_half(r);
  s[3] = r - s[2];
}
__device__ __forceinline__ void half_slices(double x, float c0, float c1, float* s) {
  s[0] = round_grid((float)x, c0);
  double r = x - (double)s[0];
  s[1] = round_grid((float)r, c1);
  r -= (double)s[1];
  s[2] = round_half((float)r);
  s[3] = (float)(r - (double)s[2]);
}
// The rounding constants of the first two slices of rows (side 0) or columns.
__device__ __forceinline__ float half_c0(int64_t k, int side) {
  return 1.5f * __int_as_float((23 + kHalfUp - first_bits(k, side) + 127) << 23);
}
__device__ __forceinline__ float half_c1(int64_t k, int side) {
  return half_c0(k, side) * __int_as_float((127 - second_bits(k)) << 23);
}
// A slice as the 16-bit operand value (exact, kHalf's last slice rounded).
template <int S>
__device__ __forceinline__ uint16_t slice_bits(float v) {
  if constexpr (Sl<S>::half) return __half_as_ushort(__float2half_rn(v));
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// 2^k as a float for -126 <= k <= 127.
__device__ __forceinline__ float pow2f(int k) { return __int_as_float((k + 127) << 23); }
// Two factors whose product is 2^-e (|e| <= 252), each a normal float: x 2^-e
// is (x f.x) f.y, exact unless the result underflows (far below any slice).
__device__ __forceinline__ float2 inv_scale(int e) {
  const int a = (-e) / 2;
  return make_float2(pow2f(a), pow2f(-e - a));
}
// x 2^-e: complex64 rows (|e| <= 149) by the two factors f, complex128 rows
// (any exponent) by ldexp.
__device__ __forceinline__ float scale_row(float x, int, float2 f) { return (x * f.x) * f.y; }
__device__ __forceinline__ double scale_row(double x, int e, float2) { return ldexp(x, -e); }

// One plane tile (ROWS x 16) is shared by PARTS blocks (blockIdx.x = kt PARTS
// + part), each slicing TILE / PARTS values: complex128 B is sliced in FP64,
// whose GB300 rate is low, so the work is spread over many SMs.
template <int ROWS>
__host__ __device__ constexpr int pack_parts() {
  return ROWS * TK / 256 > 0 ? ROWS * TK / 256 : 1;
}
template <typename T, int ROWS, int S>
__global__ void __launch_bounds__(256) k_oz_pack(const T* __restrict__ X, uint16_t* __restrict__ planes,
                                                 const __grid_constant__ GemmDesc d, int side, int64_t rows,
                                                 int64_t rtiles, int64_t ktiles, const int* __restrict__ e_in) {
  constexpr int TILE = ROWS * TK, GROUPS = ROWS / 8, PARTS = pack_parts<ROWS>(), PER = TILE / PARTS, NSL = Sl<S>::n;
  __shared__ int64_t roff[ROWS];
  __shared__ int rexp[ROWS];
  __shared__ int64_t koff[TK];
  const int64_t kt = blockIdx.x / PARTS, rt = blockIdx.y, z = blockIdx.z;
  const int part = (int)(blockIdx.x % PARTS);
  const int nrm = side == 0 ? d.nm : d.nn;
  const int64_t* rdim = side == 0 ? d.mdim : d.ndim;
  const int64_t* rstr = side == 0 ? d.msa : d.nsb;
  const int64_t* kstr = side == 0 ? d.ksa : d.ksb;
  const int64_t* zstr = side == 0 ? d.zsa : d.zsb;
  for (int t = threadIdx.x; t < ROWS + TK; t += blockDim.x) {
    if (t < ROWS) {
      const int64_t r = rt * ROWS + t;
      roff[t] = r < rows ? decode(r, nrm, rdim, rstr) : -1;
      rexp[t] = r < rows ? e_in[z * rows + r] : kExpZero;
    } else {
      const int64_t k = kt * TK + (t - ROWS);
      koff[t - ROWS] = k < d.K ? decode(k, d.nk, d.kdim, kstr) : -1;
    }
  }
  __syncthreads();
  const int64_t zo = decode(z, d.nz, d.zdim, zstr);
  using R = typename Real<T>::R;
  uint16_t* tile = planes + (((z * rtiles + rt) * ktiles + kt) * Sl<S>::planes) * (int64_t)TILE;
  const float c0 = half_c0(d.K, side), c1 = half_c1(d.K, side);
  for (int o = part * PER + threadIdx.x; o < (part + 1) * PER; o += blockDim.x) {
    // o = ((kc * GROUPS + g) * 8 + r8) * 8 + k8: core matrix (kc, g), row r8, K k8
    const int core = o >> 6, within = o & 63;
    const int kc = core / GROUPS, g = core - kc * GROUPS;
    const int r = g * 8 + (within >> 3), k = kc * 8 + (within & 7);
    float re[NSL], im[NSL];
#pragma unroll
    for (int i = 0; i < NSL; ++i) re[i] = im[i] = 0.f;
    if (roff[r] >= 0 && koff[k] >= 0 && rexp[r] != kExpZero) {
      const T v = X[zo + roff[r] + koff[k]];
      if constexpr (Sl<S>::half) {
        half_slices(scale2((R)v.x, kHalfUp - rexp[r]), c0, c1, re);
        half_slices(scale2((R)v.y, kHalfUp - rexp[r]), c0, c1, im);
      } else {
        slices<R, NSL>(scale2((R)v.x, -rexp[r]), re);
        slices<R, NSL>(scale2((R)v.y, -rexp[r]), im);
      }
    }
    if constexpr (ROWS == 16) {
      // 16-wide tiles: per part (Re, Im) one block of the NSL slices side by
      // side along N (slice i = rows 16 i .. 16 i + 15, row groups 2 i and
      // 2 i + 1), so that slices 0 .. m form one operand of 16 (m + 1) rows
      const int r8 = within >> 3, k8 = within & 7;
#pragma unroll
      for (int i = 0; i < NSL; ++i) {
        const int q = ((kc * (NSL * GROUPS) + i * GROUPS + g) * 8 + r8) * 8 + k8;
        tile[0 * NSL * TILE + q] = slice_bits<S>(re[i]);
        tile[1 * NSL * TILE + q] = slice_bits<S>(im[i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NSL; ++i) {
        tile[(0 * NSL + i) * TILE + o] = slice_bits<S>(re[i]);
        tile[(1 * NSL + i) * TILE + o] = slice_bits<S>(im[i]);
      }
    }
  }
}

constexpr int kParkPitch = 132;  // floats per parked row: 16-byte accesses of eight rows on different banks
// A column of the tile being stored, for the epilogue of parked sums: byte
// offset in C and scale exponent, read by a warp at a time as one broadcast.
struct alignas(16) ParkCol {
  long long off;
  int eb, pad;
};

template <int TN, int S, bool PARK>
struct alignas(1024) OzSmem {
  unsigned char a[OzCfg<TN, S, PARK>::a_stages][OzCfg<TN, S, PARK>::a_bytes];  // ring of A stacks
  unsigned char b[OzCfg<TN, S, PARK>::b_stages][OzCfg<TN, S, PARK>::b_bytes];  // ring of B planes
  int64_t koff[kMaxK];                                                        // A's K offsets
  uint64_t full_a[OzCfg<TN, S, PARK>::a_stages];
  uint64_t empty_a[OzCfg<TN, S, PARK>::a_stages];
  uint64_t full_b[OzCfg<TN, S, PARK>::one_ring ? 1 : OzCfg<TN, S, PARK>::b_stages];
  uint64_t empty_b[OzCfg<TN, S, PARK>::one_ring ? 1 : OzCfg<TN, S, PARK>::b_stages];
  uint64_t accf[2];  // accumulator set b holds a finished tile
  uint64_t acce[2];  // the epilogue has read accumulator set b
  uint64_t drain;
  uint32_t tmem_base;
  alignas(16) float park[PARK ? 2 * kRows * kParkPitch : 1];  // [Re, Im][row][column] sums of a tile
  ParkCol cols[PARK ? TN : 1];
};

// a + b = s + e exactly (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float a, float b, float& e) {
  const float s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
  return s;
}
// (l0 + l1 + l2) rounded once (before scaling): l0 + l1 by an error-free
// two-sum, the small l2 added to its error term.
__device__ __forceinline__ float level_sum(float l0, float l1, float l2) {
  float e;
  const float s = two_sum(l0, l1, e);
  return s + (e + l2);
}
// x 2^ex with one rounding, the same value as ldexpf(x, ex): a multiply by an
// exact power of two when 2^ex is a normal float.
__device__ __forceinline__ float scale_pow2(float x, int ex) {
  return (ex >= -126 && ex <= 127) ? x * __int_as_float((ex + 127) << 23) : ldexpf(x, ex);
}
__device__ __forceinline__ float combine(float l0, float l1, float l2, int ex, float) {
  return scale_pow2(level_sum(l0, l1, l2), ex);
}
__device__ __forceinline__ double combine(float l0, float l1, float l2, int ex, double) {
  return ldexp(((double)l0 + (double)l1) + (double)l2, ex);
}

// Two slice values (k, k + 1) as one 32-bit word of 16-bit operands.
template <int S>
__device__ __forceinline__ uint32_t pack_x2(float lo, float hi) {
  if constexpr (Sl<S>::half) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // exact: slices have <= 8 bits
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// A values per converter thread and K tile: 8 for complex64 A (whole 16-byte
// core-matrix rows), 4 for complex128 A.
template <typename TA>
__host__ __device__ constexpr int conv_values() {
  return sizeof(TA) == 8 ? 8 : 4;
}
// Generic-proxy shared-memory writes made visible to the tensor core's reads.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// True when `v` holds in every thread of the epilogue warps, all of which call
// it (named barrier 1, 8 warps; shared-memory accesses before it are seen after it).
__device__ __forceinline__ bool epilogue_all(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n barrier.cta.red.and.pred p, 1, %2, q;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "n"(32 * 8)
      : "memory");
  return r != 0;
}

// The ring position `by` stages on (by <= kStages), with its phase.
template <int kStages>
__device__ __forceinline__ void next_stage(int& s, uint32_t& ph, int by = 1) {
  s += by;
  if (s >= kStages) {
    s -= kStages;
    ph ^= 1u;
  }
}

template <typename TA, typename TC, int TN, int S, int CONV>
__global__ void __launch_bounds__(kThreads, 1)
    k_oz_gemm(const TA* __restrict__ A, const uint16_t* __restrict__ pb, TC* __restrict__ C,
              const __grid_constant__ GemmDesc d, const int64_t* __restrict__ cm_tab,
              const int64_t* __restrict__ cn_tab, const int* __restrict__ ea, const int* __restrict__ eb,
              int64_t mtiles, int64_t ntiles, int64_t ktiles, int kvec, int* status) {
  constexpr bool kPark = oz_park<TC, TN, S>();
  using CF = OzCfg<TN, S, kPark>;
  constexpr int kSlices = Sl<S>::n, kPlanes = Sl<S>::planes, kPairs = Sl<S>::pairs;
  constexpr int kAStages = CF::a_stages, kBStages = CF::b_stages;
  constexpr uint32_t kTmemCols = CF::tmem_cols;
  constexpr int kSets = CF::acc_sets;
  constexpr int kConvWarps = CONV, kEpiWarps = kWorkWarps - kConvWarps;
  constexpr int kGroupThreads = kRows * TK / conv_values<TA>();  // converters of one K tile
  static_assert(!kPark || kEpiWarps == 8, "epilogue_all counts 8 warps");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  OzSmem<TN, S, kPark>& sm = *reinterpret_cast<OzSmem<TN, S, kPark>*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ntot = ntiles * mtiles * d.Z;
  uint64_t* const full_b = CF::one_ring ? sm.full_a : sm.full_b;
  uint64_t* const empty_b = CF::one_ring ? sm.empty_a : sm.empty_b;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kAStages; ++s) {
      // one arrival per warp of the converter group of the K tile (and the producer's)
      mbar_init(&sm.full_a[s], kGroupThreads / 32 + (CF::one_ring ? 1 : 0));
      mbar_init(&sm.empty_a[s], 1);
    }
    if constexpr (!CF::one_ring)
      for (int s = 0; s < kBStages; ++s) {
        mbar_init(&sm.full_b[s], 1);  // the producer's expect_tx
        mbar_init(&sm.empty_b[s], 1);
      }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.accf[b], 1);
      mbar_init(&sm.acce[b], kEpiWarps);  // one arrival per epilogue warp
    }
    mbar_init(&sm.drain, 1);
    mbar_init_fence();
  }
  for (int t = threadIdx.x; t < d.K; t += blockDim.x) sm.koff[t] = decode(t, d.nk, d.kdim, d.ksa);
  if (warp == 1) tmem_alloc(&sm.tmem_base, kTmemCols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = sm.tmem_base;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      int64_t g = 0;  // K tiles issued so far (all tiles)
      for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x) {
        const int64_t nt = tile % ntiles, z = tile / (ntiles * mtiles);
        const uint16_t* btile = pb + ((z * ntiles + nt) * ktiles) * (int64_t)(kPlanes * CF::kBTile);
        for (int64_t kt = 0; kt < ktiles; ++kt, ++g) {
          const int s = (int)(g % kBStages);
          const uint32_t ph = (uint32_t)((g / kBStages) & 1);
          if (!mbar_wait(&empty_b[s], ph ^ 1)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full_b[s], CF::b_bytes);
          bulk_g2s(sm.b[s], btile + kt * (kPlanes * CF::kBTile), CF::b_bytes, &full_b[s]);
        }
      }
      // the copies of the last stages are in flight until their full barrier
      // completes: wait (bounded) so none lands after the CTA has exited
      for (int64_t i = g - 1; i >= 0 && i >= g - kBStages; --i)
        if (!mbar_wait(&full_b[i % kBStages], (uint32_t)((i / kBStages) & 1))) ok = false;
    }
  } else if (warp == 1) {
    // The whole warp runs the loop and waits, and one elected thread issues a
    // K tile's MMAs and its commit, so that descriptors and predicates stay
    // uniform: one MMA takes 64 cycles of the tensor core, and issued from a
    // lane-0 branch with 64-bit descriptor sums they came 79-81 cycles apart
    // (69 with this form).
    constexpr uint32_t idesc = idesc_f16(Sl<S>::half, 128, TN), idesc_neg = idesc_f16(Sl<S>::half, 128, TN, true);
    constexpr uint32_t ALBO = 24 * 128, BLBO = (TN / 8) * 128, SBO = 128;
    // positions in the rings of A and B, with their phases
    struct Pos {
      int a = 0, b = 0;
      uint32_t pa = 0, pb = 0;
    } at;
    auto filled = [&](const Pos& p) {
      return __all_sync(0xffffffffu, mbar_wait(&sm.full_a[p.a], p.pa) &&
                                         (CF::one_ring || mbar_wait(&full_b[p.b], p.pb)));
    };
    auto advance = [&](Pos& p) {
      next_stage<kAStages>(p.a, p.pa);
      next_stage<kBStages>(p.b, p.pb);
    };
    // both stages are free once the MMAs issued so far have finished
    auto release = [&](const Pos& p) {
      mma_commit(&sm.empty_a[p.a]);
      if constexpr (!CF::one_ring) mma_commit(&empty_b[p.b]);
    };
    int64_t t = 0;   // tiles of this CTA
    // The MMAs of the K tile at `p`, levels lo .. hi (2: the rest).  kHalf: the
    // MMAs of one A operand follow each other, the last slices first: the first
    // MMA fills the tensor core's A buffer from shared memory, the others use it
    // (an M = N = 128 MMA reads 8 KB in its 64 cycles, all of the SM's
    // shared-memory bandwidth).  bf16 slices: level by level (pair_i).  `first`
    // overwrites the levels; l2 is the column of level 2.
    auto issue = [&](const Pos& p, int lo, int hi, bool first, uint32_t set, uint32_t l2) {
      const uint32_t sa = smem_u32(sm.a[p.a]) >> 4, sb = smem_u32(sm.b[p.b]) >> 4;
      // part 0: [Ar; Ai] . Br = [Ar.Br ; Ai.Br]; part 1: [Ai; -Ar] with A
      // negated . Bi = [-Ai.Bi ; Ar.Bi]
      auto adesc = [&](int i, int part) { return desc_at(sa + ((i * kStackBytes + part * 8 * 128) >> 4), ALBO, SBO); };
      auto bdesc = [&](int j, int part) {
        return desc_at(sb + (((part * kSlices + j) * CF::kBTile * 2) >> 4), BLBO, SBO);
      };
      auto level = [&](int lv) { return tmem + (lv < 2 ? set + (uint32_t)(lv * TN) : l2); };
      if constexpr (Sl<S>::half) {
#pragma unroll
        for (int i = kSlices - 1; i >= 0; --i) {
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            const uint64_t x = adesc(i, part);
            const int j0 = i >= lo ? 0 : lo - i;  // B's slices j1 - 1 .. j0
            const int j1 = hi < 2 && Sl<S>::met(i) > hi + 1 - i ? hi + 1 - i : Sl<S>::met(i);
#pragma unroll
            for (int j = Sl<S>::met(0) - 1; j >= 0; --j) {
              if (j < j0 || j >= j1) continue;
              // the first MMA into each level, pairs (0,0), (1,0) and (3,0), overwrites it
              const uint32_t acc = (first && part == 0 && j == 0 && i != 2) ? 0u : 1u;
              const uint32_t dl = level(i + j);
              const uint64_t y = bdesc(j, part);
              const uint32_t id = part ? idesc_neg : idesc;
              if (j == j1 - 1)
                mma_f16_a_fill(dl, x, y, id, acc);
              else if (j > j0)
                mma_f16_a_use(dl, x, y, id, acc);
              else
                mma_f16_a_lastuse(dl, x, y, id, acc);
            }
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
          const int i = pair_i<S>(q), j = pair_j<S>(q), lv = i + j < 2 ? i + j : 2;
          if (lv < lo || lv > hi) continue;
          // the first pair of each level overwrites it
          mma_f16(level(lv), adesc(i, 0), bdesc(j, 0), idesc, first && (q < 2 || q == 3) ? 0u : 1u);
          mma_f16(level(lv), adesc(i, 1), bdesc(j, 1), idesc_neg, 1u);
        }
      }
    };
    for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x, ++t) {
      const int b = (int)(t % kSets);
      int kt0 = 0;  // K tiles whose MMAs are all issued
      if constexpr (kPark) {
        // Level 2 alternates between TMEM blocks 2 and 3, so the first K tiles'
        // level-2 MMAs (16 of 22) do not wait for the epilogue of the tile
        // before; their level 0 and 1 MMAs follow once it has read its sums.
        const uint32_t l2 = (uint32_t)((2 + (t & 1)) * TN);
        static_assert(kAStages <= kBStages, "K tiles issued ahead");
        const int pre = (int)ktiles < kAStages ? (int)ktiles : kAStages;
        Pos ahead = at;
        for (int kt = 0; kt < pre && ok; ++kt) {
          if (!filled(ahead)) ok = false;
          fence_after();
          if (ok && elect_one()) issue(ahead, 2, 2, kt == 0, 0, l2);
          __syncwarp();
          advance(ahead);
        }
        if (!ok || !__all_sync(0xffffffffu, mbar_wait(&sm.acce[b], (uint32_t)((t & 1) ^ 1)))) {
          ok = false;
          break;
        }
        fence_after();
        for (int kt = 0; kt < pre; ++kt) {
          if (elect_one()) {
            issue(at, 0, 1, kt == 0, 0, l2);
            release(at);
          }
          __syncwarp();
          advance(at);
        }
        kt0 = pre;
      } else {
        // the epilogue has read this accumulator set's previous tile
        if (!__all_sync(0xffffffffu, mbar_wait(&sm.acce[b], (uint32_t)(((t / kSets) & 1) ^ 1)))) {
          ok = false;
          break;
        }
        fence_after();
      }
      for (int kt = kt0; kt < (int)ktiles; ++kt) {
        if (!filled(at)) {
          ok = false;
          break;
        }
        fence_after();
        if constexpr (CF::narrow) {
          const uint32_t sa = smem_u32(sm.a[at.a]) >> 4, sb = smem_u32(sm.b[at.b]) >> 4;
          // B block per part: the slices x 2 row groups per K half
          constexpr uint32_t NLBO = kSlices * 2 * 128;
          if (elect_one()) {
#pragma unroll
            for (int i = 0; i < kSlices; ++i) {
              const uint32_t dl = tmem + (uint32_t)(b * CF::set_cols + narrow_col<S>(i));
              const uint64_t x1 = desc_at(sa + ((i * kStackBytes) >> 4), ALBO, SBO);            // [Ar; Ai]
              const uint64_t x2 = desc_at(sa + ((i * kStackBytes + 8 * 128) >> 4), ALBO, SBO);  // [Ai; -Ar]
              const uint64_t br = desc_at(sb, NLBO, SBO);
              const uint64_t bi = desc_at(sb + ((kSlices * CF::kBTile * 2) >> 4), NLBO, SBO);
              // [Ar.Br ; Ai.Br], then [-Ai.Bi ; Ar.Bi], slices 0 .. met(i)-1 of B
              mma_f16(dl, x1, br, idesc_f16(Sl<S>::half, 128, 16 * Sl<S>::met(i)), kt == 0 ? 0u : 1u);
              mma_f16(dl, x2, bi, idesc_f16(Sl<S>::half, 128, 16 * Sl<S>::met(i), true), 1u);
            }
            release(at);
          }
          __syncwarp();
          advance(at);
          continue;
        }
        if (elect_one()) {
          if constexpr (kPark)
            issue(at, 0, 2, false, 0, (uint32_t)((2 + (t & 1)) * TN));
          else
            issue(at, 0, 2, kt == 0, (uint32_t)(b * 3 * TN), (uint32_t)((b * 3 + 2) * TN));
          release(at);
        }
        __syncwarp();
        advance(at);
      }
      if (!ok) break;
      if (elect_one()) mma_commit(&sm.accf[b]);  // tile accumulators ready for the epilogue
    }
    // every MMA issued has finished once this arrives (TMEM is freed below)
    if (elect_one()) mma_commit(&sm.drain);
    if (!mbar_wait(&sm.drain, 0)) ok = false;
  } else if (warp < 2 + kConvWarps) {
    // converters: with NV values per thread and K tile, the converter warps
    // form groups of 64 16 / NV threads that take K tiles in turn; thread ch of a group
    // handles row r = ch % 64 and the NV consecutive K values from
    // kq = (ch / 64) NV of its K tiles.  Complex64 A: NV = 8, a whole 16-byte
    // core-matrix row per stack block, stored without bank conflicts;
    // complex128 A: NV = 4 (half rows; fewer registers), one group.
    constexpr int NV = conv_values<TA>(), GT = kGroupThreads, H = 32 * kConvWarps / GT;
    static_assert(H <= kAStages, "ring");
    const int c = threadIdx.x - 64;
    const int grp = c / GT, ch = c % GT;
    const int r = ch & (kRows - 1), kq = (ch >> 6) * NV;
    using R = typename Real<TA>::R;
    // byte offset of (slice 0, block 0, row r, K value kq) in the stacks
    const uint32_t row_off = (uint32_t)((((kq >> 3) * 24 + (r >> 3)) * 8 + (r & 7)) * 16 + (kq & 7) * 2);
    const float hc0 = half_c0(d.K, 0), hc1 = half_c1(d.K, 0);
    // This CTA's K tiles form one sequence g = tile number * ktiles + kt; the
    // group takes g = grp, grp + H, ...  The next one's A values and row
    // exponent are loaded while this one is sliced, across tile boundaries
    // (a tile's rows and exponent are looked up once per tile).
    const int64_t ntl = blockIdx.x < ntot ? (ntot - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int64_t items = ntl * ktiles;
    const TA* prow = A;
    bool pm = false;
    int en = kExpZero;  // exponent of the prefetched K tile's row (a load in flight)
    auto row_info = [&](int64_t tl) {
      const int64_t tile = blockIdx.x + tl * gridDim.x;
      const int64_t rr = tile / ntiles, mt = rr % mtiles, z = rr / mtiles;
      const int64_t m = mt * kRows + r;
      pm = m < d.M;
      en = pm ? ea[z * d.M + m] : kExpZero;
      prow = A + (pm ? decode(z, d.nz, d.zdim, d.zsa) + decode(m, d.nm, d.mdim, d.msa) : 0);
    };
    // zeros past the operand (and for rows outside it); an all-zero row's
    // values are zeros themselves, whatever its exponent
    auto load = [&](int64_t kt, TA* v) {
      if constexpr (NV == 8) {
        if (kvec) {  // every four values from a multiple of 4 are 32 aligned bytes
          const int64_t k = kt * TK + kq;
#pragma unroll
          for (int q = 0; q < NV; q += 4) {
            if (pm && k + q < d.K) {
              ldg256(prow + sm.koff[k + q], reinterpret_cast<float*>(v + q));
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u) v[q + u].x = v[q + u].y = 0;
            }
          }
          return;
        }
      }
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const int64_t k = kt * TK + kq + q;
        if (pm && k < d.K) {
          v[q] = prow[sm.koff[k]];
        } else {
          v[q].x = 0;
          v[q].y = 0;
        }
      }
    };
    TA nxt[NV];
    // the next K tile to load: tile ptl (number within this CTA) and its K
    // tile pkt, stepped without divisions
    int64_t ptl = 0;
    int pkt = grp;
    auto settle = [&]() {
      bool moved = false;
      while (pkt >= (int)ktiles) {
        pkt -= (int)ktiles;
        ++ptl;
        moved = true;
      }
      return moved;
    };
    if (grp < items) {
      settle();
      row_info(ptl);
      load(pkt, nxt);
    }
    int s = grp;
    uint32_t ph = 0;
    for (int64_t gk = grp; gk < items && ok; gk += H) {
      const int e = en;
      TA cur[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) cur[q] = nxt[q];
      if (gk + H < items) {  // in flight while this K tile is sliced
        pkt += H;
        if (settle()) row_info(ptl);
        load(pkt, nxt);
      }
      const int up = Sl<S>::half ? kHalfUp : 0;
      const float2 f = inv_scale((e != kExpZero ? e : 0) - up);
      {
        uint32_t pr[kSlices][NV / 2], pim[kSlices][NV / 2];  // 16-bit pairs (k, k + 1) of Ar, Ai
#pragma unroll
        for (int q = 0; q < NV; q += 2) {
          float a0[kSlices], b0[kSlices], a1[kSlices], b1[kSlices];
          if constexpr (Sl<S>::half) {
            half_slices(scale_row((R)cur[q].x, e - up, f), hc0, hc1, a0);
            half_slices(scale_row((R)cur[q].y, e - up, f), hc0, hc1, b0);
            half_slices(scale_row((R)cur[q + 1].x, e - up, f), hc0, hc1, a1);
            half_slices(scale_row((R)cur[q + 1].y, e - up, f), hc0, hc1, b1);
          } else {
            slices<R, kSlices>(scale_row((R)cur[q].x, e, f), a0);
            slices<R, kSlices>(scale_row((R)cur[q].y, e, f), b0);
            slices<R, kSlices>(scale_row((R)cur[q + 1].x, e, f), a1);
            slices<R, kSlices>(scale_row((R)cur[q + 1].y, e, f), b1);
          }
#pragma unroll
          for (int i = 0; i < kSlices; ++i) {
            pr[i][q / 2] = pack_x2<S>(a0[i], a1[i]);
            pim[i][q / 2] = pack_x2<S>(b0[i], b1[i]);
          }
        }
        bool got = mbar_wait(&sm.empty_a[s], ph ^ 1);
        got = __all_sync(0xffffffffu, got);
        if (!got) {
          ok = false;
          break;
        }
        const uint32_t base = smem_u32(sm.a[s]) + row_off;
#pragma unroll
        for (int i = 0; i < kSlices; ++i) {
          const uint32_t slice = base + (uint32_t)(i * kStackBytes);
          constexpr uint32_t kNeg = 0x80008000u;
          if constexpr (NV == 8) {
            sts128(slice, pr[i][0], pr[i][1], pr[i][2], pr[i][3]);                              // Ar
            sts128(slice + 8 * 128, pim[i][0], pim[i][1], pim[i][2], pim[i][3]);                // Ai
            sts128(slice + 16 * 128, pr[i][0] ^ kNeg, pr[i][1] ^ kNeg, pr[i][2] ^ kNeg, pr[i][3] ^ kNeg);  // -Ar
          } else {
            sts64(slice, pr[i][0], pr[i][1]);                        // Ar
            sts64(slice + 8 * 128, pim[i][0], pim[i][1]);            // Ai
            sts64(slice + 16 * 128, pr[i][0] ^ kNeg, pr[i][1] ^ kNeg);  // -Ar
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full_a[s]);
        next_stage<kAStages>(s, ph, H);
      }
    }
  } else {
    // epilogue: warp w reads TMEM lanes of quadrant w % 4 (0, 1: Cr of rows
    // 0..63; 2, 3: Ci), columns [h TN/2, (h+1) TN/2)
    constexpr int CW = TN / (kEpiWarps / 4);
    const int q = warp & 3, h = (warp - 2 - kConvWarps) >> 2;
    const int part = q >> 1;               // 0: real parts, 1: imaginary parts
    const int r = (q & 1) * 32 + lane;     // complex row within the tile
    const uint32_t lane_base = tmem + ((uint32_t)(q * 32) << 16);
    using R = typename std::conditional<std::is_same<TC, double2>::value, double, float>::type;
    R* Cr = reinterpret_cast<R*>(C);
    constexpr int PW = CW >= 16 && !CF::narrow ? 16 : 8;   // columns per TMEM load
    // One accumulator set and complex64 results: the combined levels are
    // parked in the unused fourth TMEM block so that the accumulators are
    // released before the scaling and the scattered stores.
    constexpr bool kStash = !kPark && kSets == 1 && std::is_same<TC, float2>::value && 4 * TN <= (int)kTmemCols &&
                            CW % 16 == 0;
    // Where a thread's stores lie: its TMEM row and columns, or with parked
    // sums row half e & 1 and 32 columns from (e >> 1) 32 for epilogue warp e,
    // real and imaginary part together.
    const int e = warp - 2 - kConvWarps;
    constexpr int SW = kPark ? 32 : CW;
    const int srow = kPark ? (e & 1) * 32 + lane : r, scol = kPark ? (e >> 1) * 32 : h * CW;
    constexpr int NU = (SW + 31) / 32;       // columns of the warp's range per lane
    // per-tile offsets and scales, loaded one tile ahead: the row's from
    // this lane, the warp's columns spread over the lanes
    struct Meta {
      int64_t base, c0;
      int exa;
      bool mrow;
      int ebl[NU];
      long long cnl[NU];
    };
    auto meta = [&](int64_t tile, Meta& M) {
      const int64_t nt = tile % ntiles, rr = tile / ntiles, mt = rr % mtiles, z = rr / mtiles;
      const int64_t m = mt * kRows + srow;
      M.mrow = m < d.M;
      M.base = M.mrow ? decode(z, d.nz, d.zdim, d.zsc) + cm_tab[m] : 0;
      M.exa = M.mrow ? ea[z * d.M + m] : kExpZero;
      M.c0 = nt * TN + scol;
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int64_t col = M.c0 + lane + 32 * u;
        const bool valid = lane + 32 * u < SW && col < d.N;
        M.ebl[u] = valid ? eb[z * d.N + col] : kExpZero;
        M.cnl[u] = valid ? (long long)cn_tab[col] : 0;
      }
    };
    Meta nm;
    if (blockIdx.x < ntot) meta(blockIdx.x, nm);
    int64_t t = 0;
    for (int64_t tile = blockIdx.x; tile < ntot && ok; tile += gridDim.x, ++t) {
      const Meta M = nm;
      if (tile + gridDim.x < ntot) meta(tile + gridDim.x, nm);  // in flight during this tile
      const bool mrow = M.mrow;
      const int64_t base = M.base, c0 = M.c0;
      const int exa = M.exa;
      constexpr int kDown = Sl<S>::half ? 2 * kHalfUp : 0;  // both operands' factor, taken off
      const int b = (int)(t % kSets);
      bool got = mbar_wait(&sm.accf[b], (uint32_t)((t / kSets) & 1));
      got = __all_sync(0xffffffffu, got);  // the TMEM loads below are warp-collective
      // (with parked sums, of all epilogue warps: they meet in the barriers
      // below, and here the last tile's parked sums have been read)
      if constexpr (kPark) got = epilogue_all(got);
      if (!got) {
        ok = false;
        break;
      }
      fence_after();
      if constexpr (kPark) {
        // Phase 1 (holds levels 0 and 1): the three levels of each element
        // summed into one float in shared memory; then the accumulators are
        // released.
        float* P = sm.park + (part * kRows + r) * kParkPitch + h * CW;
        const uint32_t l2 = (uint32_t)((2 + (t & 1)) * TN);
#pragma unroll
        for (int piece = 0; piece < CW / 16; ++piece) {
          __syncwarp();
          const uint32_t col = lane_base + (uint32_t)(h * CW + piece * 16);
          float l0[16], l1[16], lr[16];
          tmem_ld16(col, l0);
          tmem_ld16(col + TN, l1);
          tmem_ld16(col + l2, lr);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            *(float4*)(P + piece * 16 + j) =
                make_float4(level_sum(l0[j], l1[j], lr[j]), level_sum(l0[j + 1], l1[j + 1], lr[j + 1]),
                            level_sum(l0[j + 2], l1[j + 2], lr[j + 2]), level_sum(l0[j + 3], l1[j + 3], lr[j + 3]));
        }
        if (!(e & 1)) sm.cols[scol + lane] = ParkCol{M.cnl[0] * (long long)sizeof(float2), M.ebl[0], 0};
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acce[b]);
        epilogue_all(true);  // the sums of both parts are parked
        // Phase 2 (overlaps the next tile's MMAs): scale by 2^(ea + eb), store
        // whole complex values through the result index map.
        const float* Re = sm.park + srow * kParkPitch + scol;
        const float* Im = Re + kRows * kParkPitch;
        const ParkCol* cols = sm.cols + scol;
        char* Crow = reinterpret_cast<char*>(C + base);
        const int ncol = (int)(d.N - c0 < SW ? d.N - c0 : SW);
        // Whole column ranges whose scales are normal floats in every row go
        // without a branch, so that the columns' loads and stores overlap: with
        // two branches per column (zero row, scale outside the normal range)
        // this phase took 275 cycles per column and 82 % of a tile of one K tile
        // (2^20 x 256 x 16 with the exponent pass, 8 products: 1.31 -> 0.77 ms).
        const int emin = __reduce_min_sync(0xffffffffu, M.ebl[0]), emax = __reduce_max_sync(0xffffffffu, M.ebl[0]);
        const bool plain = !mrow || (exa + emin - kDown >= -126 && exa + emax - kDown <= 127);
        if (__all_sync(0xffffffffu, plain && ncol == SW)) {
          const int ef = exa - kDown + 127;
#pragma unroll 2
          for (int cc = 0; cc < SW; cc += 4) {
            const float4 re = *(const float4*)(Re + cc), im = *(const float4*)(Im + cc);
            const ParkCol q0 = cols[cc], q1 = cols[cc + 1], q2 = cols[cc + 2], q3 = cols[cc + 3];
            const float f0 = __int_as_float((ef + q0.eb) << 23), f1 = __int_as_float((ef + q1.eb) << 23),
                        f2 = __int_as_float((ef + q2.eb) << 23), f3 = __int_as_float((ef + q3.eb) << 23);
            if (mrow) {
              *(float2*)(Crow + q0.off) = make_float2(re.x * f0, im.x * f0);
              *(float2*)(Crow + q1.off) = make_float2(re.y * f1, im.y * f1);
              *(float2*)(Crow + q2.off) = make_float2(re.z * f2, im.z * f2);
              *(float2*)(Crow + q3.off) = make_float2(re.w * f3, im.w * f3);
            }
          }
        } else {
#pragma unroll 1
          for (int cc = 0; cc < ncol; ++cc) {
            const ParkCol col = cols[cc];
            const int ex = exa + col.eb - kDown;
            const bool zero = exa == kExpZero || ex < -2 * 1100;
            if (mrow)
              *(float2*)(Crow + col.off) =
                  zero ? make_float2(0.f, 0.f) : make_float2(scale_pow2(Re[cc], ex), scale_pow2(Im[cc], ex));
          }
        }
        continue;
      }
      if constexpr (kStash) {
        // Phase 1 (holds the accumulators): the three levels of each element
        // summed into one float, parked in the spare TMEM block (columns
        // 3 TN .. 4 TN, the same lanes); then the accumulators are released.
#pragma unroll
        for (int piece = 0; piece < CW / 16; ++piece) {
          __syncwarp();
          const uint32_t col = (uint32_t)(h * CW + piece * 16);
          float l0[16], l1[16], l2[16];
          tmem_ld16(lane_base + col + 0 * TN, l0);
          tmem_ld16(lane_base + col + 1 * TN, l1);
          tmem_ld16(lane_base + col + 2 * TN, l2);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) l0[j] = level_sum(l0[j], l1[j], l2[j]);
          tmem_st16(lane_base + 3 * TN + col, l0);
        }
        tmem_wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acce[b]);
        // Phase 2 (overlaps the next tile's MMAs): scale by 2^(ea + eb) and
        // scatter through the result index map.
#pragma unroll
        for (int piece = 0; piece < CW / 16; ++piece) {
          __syncwarp();
          float v[16];
          tmem_ld16(lane_base + 3 * TN + (uint32_t)(h * CW + piece * 16), v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int cc = piece * 16 + j;
            const int ebj = __shfl_sync(0xffffffffu, M.ebl[cc / 32], cc % 32);
            const long long cnj = __shfl_sync(0xffffffffu, M.cnl[cc / 32], cc % 32);
            if (mrow && c0 + cc < d.N) {
              const int ex = exa + ebj - kDown;
              const R val = (exa == kExpZero || ex < -2 * 1100) ? (R)0 : (R)scale_pow2(v[j], ex);
              Cr[2 * (base + cnj) + part] = val;
            }
          }
        }
        continue;
      }
#pragma unroll
      for (int piece = 0; piece < CW / PW; ++piece) {
        __syncwarp();  // the TMEM loads are warp-collective
        const uint32_t col = (uint32_t)(b * 3 * TN + h * CW + piece * PW);
        float l0[PW], l1[PW], l2[PW];
        if constexpr (CF::narrow) {
          // the slice-pair regions (each a sum over K of one pair): level 0 =
          // (0,0); level 1 = (0,1) + (1,0); the others summed in FP32, the
          // smallest first, four regions per TMEM wait
          static_assert(PW == 8, "narrow tiles: 8 columns per epilogue warp");
          const uint32_t rb = lane_base + (uint32_t)(b * CF::set_cols + h * CW + piece * PW);
          float t0[PW], t1[PW];
          tmem_ld8(rb + narrow_col<S>(0), l0);
          tmem_ld8(rb + narrow_col<S>(0) + 16, t0);
          tmem_ld8(rb + narrow_col<S>(1), t1);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < PW; ++q) {
            l1[q] = t0[q] + t1[q];
            l2[q] = 0.f;
          }
#pragma unroll
          for (int p0 = 3; p0 < kPairs; p0 += 4) {
            float tb[4][PW];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (p0 + u < kPairs) tmem_ld8(rb + narrow_col<S>(pair_i<S>(p0 + u)) + 16 * pair_j<S>(p0 + u), tb[u]);
            tmem_wait_ld();
#pragma unroll
            for (int u = 0; u < 4; ++u)
              if (p0 + u < kPairs)
#pragma unroll
                for (int q = 0; q < PW; ++q) l2[q] += tb[u][q];
          }
        } else if constexpr (PW == 16) {
          tmem_ld16(lane_base + col + 0 * TN, l0);
          tmem_ld16(lane_base + col + 1 * TN, l1);
          tmem_ld16(lane_base + col + 2 * TN, l2);
        } else {
          tmem_ld8(lane_base + col + 0 * TN, l0);
          tmem_ld8(lane_base + col + 1 * TN, l1);
          tmem_ld8(lane_base + col + 2 * TN, l2);
        }
        tmem_wait_ld();
        if (piece == CW / PW - 1) {  // every value of this tile is in registers
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.acce[b]);
        }
#pragma unroll
        for (int j = 0; j < PW; ++j) {
          const int cc = piece * PW + j;  // column within the warp's range
          const int ebj = __shfl_sync(0xffffffffu, M.ebl[cc / 32], cc % 32);
          const long long cnj = __shfl_sync(0xffffffffu, M.cnl[cc / 32], cc % 32);
          if (mrow && c0 + cc < d.N) {
            const int ex = exa + ebj - kDown;
            const R v = (exa == kExpZero || ex < -2 * 1100) ? (R)0 : combine(l0[j], l1[j], l2[j], ex, R());
            Cr[2 * (base + cnj) + part] = v;
          }
        }
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

int oz_tile_n(int64_t n) { return n <= 16 ? 16 : (n <= 32 ? 32 : (n <= 64 ? 64 : 128)); }
// Tile width of an oriented pair: the autotuner's choice when it set one,
// else the narrowest tile that covers N (at most 128).
int oz_tile_of(const GemmDesc& d) {
  return (d.tile_n == 16 || d.tile_n == 32 || d.tile_n == 64 || d.tile_n == 128) ? d.tile_n : oz_tile_n(d.N);
}

struct OzLayout {
  int tn;
  int64_t mt, nt, kt;
  size_t pb, cm, cn, ea, eb, total;  // byte offsets from the aligned base
};

OzLayout layout(const GemmDesc& d, int nsl) {
  OzLayout L;
  L.tn = oz_tile_of(d);
  L.mt = ceil_div(d.M, kRows);
  L.nt = ceil_div(d.N, L.tn);
  L.kt = ceil_div(d.K, TK);
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  L.pb = 0;
  L.cm = up(L.pb + (size_t)(d.Z * L.nt * L.kt) * (2 * nsl) * (L.tn * TK) * 2);
  L.cn = up(L.cm + (size_t)d.M * 8);
  L.ea = up(L.cn + (size_t)d.N * 8);
  L.eb = up(L.ea + (size_t)(d.Z * d.M) * 4);
  L.total = up(L.eb + (size_t)(d.Z * d.N) * 4) + 256;
  return L;
}

// The kernels keep the long side on M (the TMEM lanes): a pair whose A side
// is the narrow one is run as C = B x A with the roles swapped.
GemmDesc swapped(const GemmDesc& d) {
  GemmDesc s = d;
  s.M = d.N;
  s.N = d.M;
  s.nm = d.nn;
  s.nn = d.nm;
  for (int i = 0; i < kMaxModes; ++i) {
    s.mdim[i] = d.ndim[i];
    s.msa[i] = d.nsb[i];
    s.msc[i] = d.nsc[i];
    s.ndim[i] = d.mdim[i];
    s.nsb[i] = d.msa[i];
    s.nsc[i] = d.msc[i];
    s.ksa[i] = d.ksb[i];
    s.ksb[i] = d.ksa[i];
    s.zsa[i] = d.zsb[i];
    s.zsb[i] = d.zsa[i];
  }
  return s;
}
// Orientation: the autotuner's choice (orient 1 = as given, 2 = swapped) when
// it set one, else swap when A is the narrow side.
bool needs_swap(const GemmDesc& d) {
  if (d.orient == 1) return false;
  if (d.orient == 2) return true;
  return d.M < 64 && d.N > d.M;
}

// B's column exponents (16 columns per block, 16 threads on each: B is the
// small side, so its pass needs many blocks to be short), then its slices.
template <typename T, int ROWS, int S>
void prep_b(const void* X, uint16_t* planes, int* e, const GemmDesc& d, int64_t rtiles, int64_t kt,
            cudaStream_t s) {
  k_oz_exp<T, 16><<<dim3((unsigned)ceil_div(d.N, 16), (unsigned)d.Z), 256, 0, s>>>((const T*)X, d, 1, d.N, e);
  constexpr int parts = pack_parts<ROWS>();
  k_oz_pack<T, ROWS, S><<<dim3((unsigned)(kt * parts), (unsigned)rtiles, (unsigned)d.Z), 256, 0, s>>>(
      (const T*)X, planes, d, 1, d.N, rtiles, kt, e);
}

template <typename T, int S>
void prep_b_tn(const void* X, int tn, uint16_t* planes, int* e, const GemmDesc& d, int64_t rtiles, int64_t kt,
               cudaStream_t s) {
  if (tn == 128) prep_b<T, 128, S>(X, planes, e, d, rtiles, kt, s);
  else if (tn == 64) prep_b<T, 64, S>(X, planes, e, d, rtiles, kt, s);
  else if (tn == 32) prep_b<T, 32, S>(X, planes, e, d, rtiles, kt, s);
  else prep_b<T, 16, S>(X, planes, e, d, rtiles, kt, s);
}

template <typename TA, typename TC, int TN, int S, int CONV>
cudaError_t oz_gemm_launch(const void* A, const uint16_t* pb, void* C, const GemmDesc& d, const int64_t* cm,
                           const int64_t* cn, const int* ea, const int* eb, const OzLayout& L, int* status,
                           cudaStream_t s) {
  constexpr bool park = oz_park<TC, TN, S>();
  static_assert(sizeof(OzSmem<TN, S, park>) + 1024 <= 232448, "shared memory layout exceeds 227 KiB");
  const size_t smem = sizeof(OzSmem<TN, S, park>) + 1024;
  static bool attr = false;
  if (!attr) {
    cudaError_t e =
        cudaFuncSetAttribute(k_oz_gemm<TA, TC, TN, S, CONV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int64_t tiles = L.mt * L.nt * d.Z;
  const unsigned grid = (unsigned)std::min<int64_t>(tiles, sm_count());
  k_oz_gemm<TA, TC, TN, S, CONV><<<grid, kThreads, smem, s>>>((const TA*)A, pb, (TC*)C, d, cm, cn, ea, eb, L.mt, L.nt,
                                                              L.kt, k_vector(A, d) ? 1 : 0, status);
  return cudaGetLastError();
}

template <typename TA, typename TC, int S>
cudaError_t oz_gemm_tn(const void* A, const uint16_t* pb, void* C, const GemmDesc& d, const int64_t* cm,
                       const int64_t* cn, const int* ea, const int* eb, const OzLayout& L, int* status,
                       cudaStream_t s) {
  if (L.tn == 128) return oz_gemm_launch<TA, TC, 128, S, 8>(A, pb, C, d, cm, cn, ea, eb, L, status, s);
  if (L.tn == 64) return oz_gemm_launch<TA, TC, 64, S, 8>(A, pb, C, d, cm, cn, ea, eb, L, status, s);
  if (L.tn == 32) return oz_gemm_launch<TA, TC, 32, S, 8>(A, pb, C, d, cm, cn, ea, eb, L, status, s);
  if (many_converters<TA, 16, S>() && L.kt > 6)
    return oz_gemm_launch<TA, TC, 16, S, many_converters<TA, 16, S>() ? 12 : 8>(A, pb, C, d, cm, cn, ea, eb, L, status, s);
  return oz_gemm_launch<TA, TC, 16, S, 8>(A, pb, C, d, cm, cn, ea, eb, L, status, s);
}

bool eligible_oriented(const GemmDesc& d) {
  if (d.M < 64 || d.N < 8 || d.K < 16 || d.K > kMaxK) return false;
  // fewer than 512 complex products per output (e.g. a tall operand absorbing
  // a 16-column gate tensor over K = 16): memory-bound work whose per-tile
  // costs here exceed a plain FP32 pass, and whose FP32 sums have <= 32 terms
  if (d.N * d.K < 512) return false;
  if (d.Z > 65535 || ceil_div(d.N, oz_tile_of(d)) > 65535) return false;  // grid y / z of the B passes
  return layout(d, 5).total <= (size_t(24) << 30);
}

}  // namespace

bool oz_eligible(const GemmDesc& d) { return eligible_oriented(needs_swap(d) ? swapped(d) : d); }

size_t oz_scratch_bytes(int slices, const GemmDesc& d) { return layout(needs_swap(d) ? swapped(d) : d, slices).total; }

template <int S, typename TC>
static cudaError_t launch_oz_n(int ta, int tb, const void* A, const void* B, void* C, const GemmDesc& d,
                               char* base, const OzLayout& L, int* status, cudaStream_t stream) {
  auto* pb = (uint16_t*)(base + L.pb);
  auto* cm = (int64_t*)(base + L.cm);
  auto* cn = (int64_t*)(base + L.cn);
  auto* ea = (int*)(base + L.ea);
  auto* eb = (int*)(base + L.eb);
  if (ta == PQ_C128)
    row_exponents((const double2*)A, d, ea, stream);
  else
    row_exponents((const float2*)A, d, ea, stream);
  if (tb == PQ_C128)
    prep_b_tn<double2, S>(B, L.tn, pb, eb, d, L.nt, L.kt, stream);
  else
    prep_b_tn<float2, S>(B, L.tn, pb, eb, d, L.nt, L.kt, stream);
  const int64_t idx_blocks = std::min<int64_t>(ceil_div(d.M + d.N, 256), 152 * 8);
  k_result_index<<<(unsigned)idx_blocks, 256, 0, stream>>>(d, cm, cn);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return ta == PQ_C128 ? oz_gemm_tn<double2, TC, S>(A, pb, C, d, cm, cn, ea, eb, L, status, stream)
                       : oz_gemm_tn<float2, TC, S>(A, pb, C, d, cm, cn, ea, eb, L, status, stream);
}

cudaError_t launch_oz(int slices, int ta, int tb, int tc, const void* A, const void* B, void* C,
                      const GemmDesc& d0, void* scratch, size_t scratch_bytes, int* status, cudaStream_t stream) {
  if (!oz_eligible(d0) || (slices != 5 && slices != 4 && slices != 3)) return cudaErrorNotSupported;
  const bool swap = needs_swap(d0);
  const GemmDesc d = swap ? swapped(d0) : d0;
  if (swap) {
    std::swap(A, B);
    std::swap(ta, tb);
  }
  const OzLayout L = layout(d, slices);
  if (!scratch || scratch_bytes < L.total) return cudaErrorInvalidValue;
  char* base = (char*)(((uintptr_t)scratch + 255) & ~(uintptr_t)255);
  // Complex64 results up to K = kHalfMaxK take the fp16 split: no less exact than
  // five bf16 slices (above), with 11 slice products instead of 15.  Past
  // that its first slices would need 7 bits on both sides and the pairs (1,3) and
  // (3,1) to drop no more than five slices do; complex128 results need the
  // five slices' order of levels, whose rest is what their caller sees.
  const bool c128 = tc == PQ_C128;
  if (slices == 5) {
    if (c128) return launch_oz_n<5, double2>(ta, tb, A, B, C, d, base, L, status, stream);
    return d.K <= kHalfMaxK ? launch_oz_n<kHalf, float2>(ta, tb, A, B, C, d, base, L, status, stream)
                            : launch_oz_n<5, float2>(ta, tb, A, B, C, d, base, L, status, stream);
  }
  if (slices == 4)
    return c128 ? launch_oz_n<4, double2>(ta, tb, A, B, C, d, base, L, status, stream)
                : launch_oz_n<4, float2>(ta, tb, A, B, C, d, base, L, status, stream);
  return c128 ? launch_oz_n<3, double2>(ta, tb, A, B, C, d, base, L, status, stream)
              : launch_oz_n<3, float2>(ta, tb, A, B, C, d, base, L, status, stream);
}

}  // namespace pq
