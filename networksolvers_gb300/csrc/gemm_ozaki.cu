// FP64-accurate GEMM on the BF16 tensor cores by exact multi-slice splitting
// (the Ozaki scheme: K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59 (2012)).
//
// Row i of A is scaled by sigma_i = 2^ceil(log2 max_k |A_ik|) and written as
//   A_ik / sigma_i = sum_{s<S} 2^{-7(s+1)} A^(s)_ik + r,  A^(s) integers, |A^(s)| <= 128,
// (round-to-nearest digits, |r| <= 2^{-7S-1}); columns of B likewise with tau_j.  Then
//   (AB)_ij = sigma_i tau_j sum_g 2^{-7(g+2)} sum_{s+t=g} (A^(s) B^(t))_ij,   g <= S-1.
// The integer slices are exact in BF16 (|A^(0)| <= 128, the others <= 64), and with g+1 <= 8
// products per group and K chunks of 384 every partial sum is an integer below
// 384 (2 x 128 x 64 + 6 x 64^2) < 2^24, so the tcgen05 FP32 accumulation of a group over a
// chunk is exact.  Drain warps add the group sums of each chunk into double-float (hi, lo)
// FP32 accumulators; the epilogue widens to FP64 and applies sigma_i tau_j, alpha and beta.
// At the end of a chunk the tensor pipe waits for the accumulators' drain, so chunks are as
// long as exactness allows: an H_eff product at bond dimension 1024 took 0.94 ms with
// chunks of 384, 0.97 with 256 and 1.07 with 128 (0.78 since the epilogue below).  With S = 6 slices the result is
// within ~2^-43 K sigma_i tau_j of A B (dropped slices and products).
//
// Kernel layout: 128 x 64 output tile per CTA, 16 drain warps (4 warpgroups, each
// owning 16 accumulator columns) + 1 TMA/MMA warp; three-stage ring of 32-wide K slabs
// holding all six slices of A and B (SWIZZLE_64B); 6 x 64 TMEM accumulator columns.
// All mbarrier waits are bounded; on time-out the CTA raises the error flag, drains its
// TMA copies (bounded), frees its TMEM and returns.
#include "chained.h"
#include "nsg_internal.h"

#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

namespace nsg {

namespace {

constexpr int BM = 128, BN = 64, BKS = 32;  // K slab: 32 bf16 = 64 bytes
constexpr int SLICE_A = BM * BKS * 2;       // 8 KB
constexpr int SLICE_B = BN * BKS * 2;       // 4 KB
constexpr int SPLIT_SLABS = 4;              // K is split over CTAs in units of 128
constexpr int CHUNK_SLABS = 12;             // K = 384 per exact chunk
constexpr int NDRAIN_WARPS = 16;
constexpr int NTHREADS = (NDRAIN_WARPS + 1) * 32;

// S slices per operand, groups g = s + t in [0, S-1] (G x 64 TMEM columns <= 512);
// S = 8 fills TMEM and leaves room for two 96 KB stages of shared memory.
template <int S_>
struct Oz {
  static constexpr int S = S_, G = S_;
  static constexpr int STAGES = S_ <= 6 ? 3 : 2;
  static constexpr int STAGE_BYTES = S * (SLICE_A + SLICE_B);
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 512;
  static_assert(G * BN <= 512, "accumulators exceed TMEM");
  static_assert(SMEM_BYTES <= 227 * 1024, "stages exceed shared memory");
};
constexpr long long kWaitLimit = 1ll << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* fail) {
  for (long long i = 0; i < kWaitLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (fail && *fail) return false;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// K-major operand, 64-byte swizzle: 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t sdesc64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)((512u >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)4u << 61;  // 64-byte swizzle
  return d;
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ---------------------------------------------------------------------------
// scales and slices of the operands of a product:
//   scale[b][r] = 2^ceil(log2 max_k |src(r, k)|) (1 for an all-zero row),
//   out[(b*S + s)][r][k] (bf16, K-major, padded with zeros)
// Work unit: 32 rows x at most 128 of K, read into shared memory with every load of the CTA
// in flight at once (16 per thread), coalesced along whichever axis is contiguous, and
// sliced from there with 16-byte stores by integer arithmetic on the numbers' bits (the
// FP64 pipe is the slow one here).  Two forms:
//  * depths below 1024: one launch for all operands of the product (up to four: the real and
//    imaginary parts of both).  A cluster of up to 8 CTAs holds 32 rows over the whole depth,
//    the row maxima meet through distributed shared memory, and each number is read once.
//  * deeper: a pass for the row maxima and one for the slices per operand (the maxima of
//    slabs of kMaxSlab, which the second pass combines).
// Measured: both operands of an eight-slice product of order 950 in 8.7 us (scale and slice
// passes per operand that read across rows: 29, in four launches), a 5120 x 1024 operand in
// 17 + 38 us (38 + 58; one launch of clusters that kept slabs of 416 in shared memory: 105).
// ---------------------------------------------------------------------------
struct OzSource {
  const double* src;
  int64_t rows, rs, ks, bs;  // element (r, k) of batch entry b at src[b bs + r rs + k ks]
  int64_t rows_p, batch;
  double* scale;
  unsigned* part;            // row maxima of the slabs (deep form)
  __nv_bfloat16* out;
  int64_t tile_end;          // 32-row tiles of this and the earlier operands
};
struct OzSources {
  OzSource op[4];
  int n;
  int64_t K, K_p;
  int slab;  // K range of a CTA, a multiple of 32
};
constexpr int kSliceThreads = 256, kSliceWarps = kSliceThreads / 32, kSliceRows = 32, kSliceK = 128;
constexpr int64_t kShallow = 1024, kMaxSlab = 512;

// position of (row, k) in the shared-memory tile: odd row stride, octets of K swizzled
__device__ __forceinline__ int slice_at(int r, int k) {
  return r * (kSliceK + 1) + ((k & ~7) | ((k ^ (k >> 3)) & 7));
}
__device__ __forceinline__ unsigned magnitude(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }

// 32 rows x len of K of one operand into `tile`; rowmax[r] takes the largest high word of
// |row r| over them (zeroed before by the caller, and valid after a barrier).
__device__ void load_slab(const OzSource& op, const double* base, int64_t r0, int64_t k0, int len, int64_t K, double* tile,
                          unsigned* rowmax) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NV = kSliceRows * kSliceK / kSliceThreads;
  double v[NV];
  if (op.ks < op.rs) {  // lanes along K: a warp takes rows warp, warp + 8, ..., four chunks of 32 each
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      const int r = warp + kSliceWarps * (x / 4), k = lane + 32 * (x % 4);
      v[x] = k < len && r0 + r < op.rows && k0 + k < K ? base[(r0 + r) * op.rs + (k0 + k) * op.ks] : 0.0;
    }
#pragma unroll
    for (int y = 0; y < NV / 4; ++y) {
      const int r = warp + kSliceWarps * y;
      unsigned m = 0;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        if (lane + 32 * x < len) tile[slice_at(r, lane + 32 * x)] = v[4 * y + x];
        m = max(m, magnitude(v[4 * y + x]));
      }
      m = __reduce_max_sync(0xffffffffu, m);
      if (lane == 0) rowmax[r] = m;
    }
  } else {  // lanes along the rows
    const bool in = r0 + lane < op.rows;
    unsigned m = 0;
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      const int k = warp + kSliceWarps * x;
      v[x] = in && k < len && k0 + k < K ? base[(r0 + lane) * op.rs + (k0 + k) * op.ks] : 0.0;
    }
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      const int k = warp + kSliceWarps * x;
      if (k < len) tile[slice_at(lane, k)] = v[x];
      m = max(m, magnitude(v[x]));
    }
    atomicMax(&rowmax[lane], m);
  }
}

// Biased exponent of a row's scale: |row| < 2^(e - 1022), e the largest biased exponent;
// scales stay normal powers of two well inside the range (a row of subnormals takes
// 2^-1000; a row that is not finite an infinite one, for which the epilogue writes NaN).
__device__ __forceinline__ unsigned scale_exponent(unsigned m) {
  const unsigned e = m >> 20;
  return m == 0 ? 1023u : e == 0x7ffu ? 0x7ffu : max(e + 1, 23u);
}

// The tile's slices: X = round(v / scale 2^{7S}) from v's bits (the 53-bit significand
// shifted by the exponents' difference, half to even), then balanced 7-bit digits
// from the low end, |d| <= 64 (the top one up to 128): X = sum_s d_s 2^{7(S-1-s)} and
// |v / scale - X 2^{-7S}| <= 2^{-7S-1}.  Lanes take octets of a row: 16-byte stores.
template <int S>
__device__ void slice_slab(const OzSource& op, int64_t b, int64_t r0, int64_t k0, int len, int64_t K_p, const double* tile,
                           const unsigned* rowexp) {
  const int noct = len / 8;
  for (int t = threadIdx.x; t < kSliceRows * noct; t += kSliceThreads) {
    const int r = t / noct, q = t % noct;
    const int re = int(rowexp[r]);
    uint32_t w[S][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const long long bits = __double_as_longlong(tile[slice_at(r, q * 8 + j)]);
      const int e = int((bits >> 52) & 0x7ff);
      const long long m = (bits & 0xfffffffffffffll) | (e ? 0x10000000000000ll : 0);
      const int sh = 52 - 7 * S - (max(e, 1) - re);  // m 2^(e - 1075) = X 2^(re - 1023 - 7S)
      const int up = min(max(sh, 1), 55);
      long long X = sh <= 0 ? m << min(-sh, 10) : (m + ((1ll << (up - 1)) - 1) + ((m >> up) & 1)) >> up;
      if (bits < 0) X = -X;
      // the low four digits and the rest in 32-bit arithmetic
      int lo = int((X + (1ll << 27)) & ((1ll << 28) - 1)) - (1 << 27);
      int hi = int((X - lo) >> 28);
#pragma unroll
      for (int s = S - 1; s >= 0; --s) {
        int& part = s >= S - 4 ? lo : hi;
        int d = part;
        if (s > 0) {
          d = ((part + 64) & 127) - 64;
          part = (part - d) >> 7;
          if (s == S - 4) hi += part;  // (the last carry out of the low digits)
        }
        // an integer of at most 128 as bf16: the upper half of its float
        const uint32_t f = __float_as_uint(__int_as_float(0x4b400000 + d) - 12582912.f);
        w[s][j / 2] = (j & 1) ? __byte_perm(w[s][j / 2], f, 0x7632) : f;
      }
    }
#pragma unroll
    for (int s = 0; s < S; ++s)
      *(uint4*)(op.out + ((size_t)(b * S + s) * op.rows_p + r0 + r) * K_p + k0 + q * 8) =
          make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
  }
}

constexpr int kTileBytes = kSliceRows * (kSliceK + 1) * 8;

template <int S>
__global__ void __launch_bounds__(kSliceThreads) oz_slice_shallow_kernel(const __grid_constant__ OzSources P) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double tile[kTileBytes / 8];
  __shared__ unsigned rowmax[kSliceRows], rowexp[kSliceRows];
  chained_start();
  const int C = int(cluster.num_blocks()), rank = int(cluster.block_rank()), tid = threadIdx.x;
  int64_t t = blockIdx.x / C;
  int o = 0;
  while (t >= P.op[o].tile_end) ++o;
  const OzSource& op = P.op[o];
  if (o > 0) t -= P.op[o - 1].tile_end;
  const int64_t rt = op.rows_p / kSliceRows, b = t / rt, r0 = (t % rt) * kSliceRows;
  const int64_t k0 = (int64_t)rank * P.slab;
  const int len = int(max(int64_t(0), min((int64_t)P.slab, P.K_p - k0)));
  if (tid < kSliceRows) rowmax[tid] = 0;
  __syncthreads();
  load_slab(op, op.src + b * op.bs, r0, k0, len, P.K, tile, rowmax);
  cluster.sync();  // every CTA's maxima are published
  if (tid < kSliceRows) {
    unsigned m = 0;
    for (int c = 0; c < C; ++c) m = max(m, *cluster.map_shared_rank(&rowmax[tid], c));
    rowexp[tid] = scale_exponent(m);
    if (rank == 0) op.scale[b * op.rows_p + r0 + tid] = __hiloint2double(int(rowexp[tid] << 20), 0);
  }
  cluster.sync();  // the peers have read this CTA's maxima; rowexp is published
  slice_slab<S>(op, b, r0, k0, len, P.K_p, tile, rowexp);
}

// blockIdx.x = 32-row tile (over the batch), blockIdx.y = its slab of kMaxSlab (MANY: the first
// of those it takes)
template <bool MANY>
__global__ void __launch_bounds__(kSliceThreads)
    oz_row_max_kernel(const __grid_constant__ OzSource op, int64_t K, int slabs) {
  __shared__ unsigned rowmax[kSliceRows];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t rt = op.rows_p / kSliceRows, b = blockIdx.x / rt, r0 = (blockIdx.x % rt) * kSliceRows;
  const double* base = op.src + b * op.bs;
  for (int slab = blockIdx.y; slab < slabs; slab += gridDim.y) {
    const int64_t k0 = slab * kMaxSlab, k1 = min(K, k0 + kMaxSlab);
    if (tid < kSliceRows) rowmax[tid] = 0;
    __syncthreads();
    if (op.ks < op.rs) {
      for (int r = warp; r < kSliceRows; r += kSliceWarps) {
        unsigned m = 0;
        if (r0 + r < op.rows)
#pragma unroll 16
          for (int64_t k = k0 + lane; k < k1; k += 32) m = max(m, magnitude(base[(r0 + r) * op.rs + k * op.ks]));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) rowmax[r] = m;
      }
    } else {
      unsigned m = 0;
      if (r0 + lane < op.rows)
#pragma unroll 16
        for (int64_t k = k0 + warp; k < k1; k += kSliceWarps)
          m = max(m, magnitude(base[(r0 + lane) * op.rs + k * op.ks]));
      atomicMax(&rowmax[lane], m);
    }
    __syncthreads();
    // (a thread clears what it has stored)
    if (tid < kSliceRows) op.part[(int64_t)slab * op.rows_p * op.batch + blockIdx.x * kSliceRows + tid] = rowmax[tid];
    if constexpr (!MANY) break;
  }
}

// blockIdx.x = 32-row tile, blockIdx.y = its slab of kSliceK (MANY: the first of those it takes)
template <int S, bool MANY>
__global__ void __launch_bounds__(kSliceThreads)
    oz_slice_deep_kernel(const __grid_constant__ OzSource op, int64_t K, int64_t K_p, int slabs) {
  __shared__ double tile[kTileBytes / 8];
  __shared__ unsigned rowmax[kSliceRows], rowexp[kSliceRows];
  const int tid = threadIdx.x;
  const int64_t rt = op.rows_p / kSliceRows, b = blockIdx.x / rt, r0 = (blockIdx.x % rt) * kSliceRows;
  if (tid < kSliceRows) {
    unsigned m = 0;
    for (int q = 0; q < slabs; ++q) m = max(m, op.part[(int64_t)q * op.rows_p * op.batch + blockIdx.x * kSliceRows + tid]);
    rowexp[tid] = scale_exponent(m);
    rowmax[tid] = 0;
    if (blockIdx.y == 0) op.scale[blockIdx.x * kSliceRows + tid] = __hiloint2double(int(rowexp[tid] << 20), 0);
  }
  for (int64_t k0 = (int64_t)blockIdx.y * kSliceK; k0 < K_p; k0 += (int64_t)gridDim.y * kSliceK) {
    const int len = int(min((int64_t)kSliceK, K_p - k0));
    __syncthreads();  // the exponents are there, and the slab before is sliced
    load_slab(op, op.src + b * op.bs, r0, k0, len, K, tile, rowmax);
    __syncthreads();
    slice_slab<S>(op, b, r0, k0, len, K_p, tile, rowexp);
    if constexpr (!MANY) break;
  }
}

struct OzEpi {
  double* C;
  int64_t ldc, sC, M, N;
  int64_t crs;  // stride between rows of C in doubles (1, or 2 for one part of complex C)
  double alpha, beta;
  const double* sa;  // row scales of A  [batch_a][Mp]
  const double* sb;  // row scales of B^T [batch_b][Np]
  int64_t Mp, Np;
  int a_batched, b_batched;
  int* err;
  // split K: grid z = batch x nsplit, split s takes K slabs [s split_slabs, ..) (whole
  // multiples of 128) and writes its scaled partial product to W[z] (M x N, column-major);
  // oz_split_reduce_kernel adds the splits in order and applies alpha and beta
  int nsplit, split_slabs;
  double* W;
  int chained;  // the slices were complete before the launch before this one
};

// exponent k of a normal power of two 2^k
__device__ __forceinline__ int pow2_exponent(double p) {
  return int((__double_as_longlong(p) >> 52) & 0x7FF) - 1023;
}
// f as a double, for a normal f or a zero: the exponent re-biased by integer arithmetic (a
// conversion is one more operation of the FP64 pipe, which holds an SM sub-partition for 64
// cycles per operation of a warp)
__device__ __forceinline__ double widen(float f) {
  const uint32_t b = __float_as_uint(f), m = (b & 0x7fffffffu) >> 3;
  const uint32_t hi = (b & 0x7f800000u) == 0 ? 0u : (b & 0x80000000u) | (m + (896u << 20));
  return __hiloint2double(int(hi), int(b << 29));
}
// (hi + lo) 2^k: one FP64 operation, the scale added to the exponent field; out of the normal
// range by two multiplications
__device__ __forceinline__ double join_pow2(float hi, float lo, int k) {
  const double v = widen(hi) + widen(lo);
  const int vh = __double2hiint(v), e = (vh >> 20) & 0x7ff;
  if (e == 0) return 0.0;  // both zero: the terms are multiples of 2^-7(S+1)
  if (e + k < 1 || e + k > 2046)
    return v * __hiloint2double((1023 + k / 2) << 20, 0) * __hiloint2double((1023 + k - k / 2) << 20, 0);
  return __hiloint2double(vh + (k << 20), __double2loint(v));
}

__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float x) {
  float s = hi + x;
  float bb = s - hi;
  float e = (hi - (s - bb)) + (x - bb);
  hi = s;
  lo += e;
}

template <int S_>
__global__ void __launch_bounds__(NTHREADS, 1)
    oz_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int nk,
                   OzEpi ep) {
  constexpr int S = Oz<S_>::S, G = Oz<S_>::G, STAGES = Oz<S_>::STAGES, STAGE_BYTES = Oz<S_>::STAGE_BYTES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ int s_exp[BM + BN];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* accfull = empty + STAGES;
  uint64_t* accempty = accfull + 1;
  uint32_t* tmem_slot = (uint32_t*)(accempty + 1);
  volatile int* fail = (volatile int*)(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int sp = int(blockIdx.z % unsigned(ep.nsplit)), bz = int(blockIdx.z / unsigned(ep.nsplit));
  const int tb = sp * ep.split_slabs;           // this split's first K slab (global index)
  const int nkl = min(nk - tb, ep.split_slabs);  // its slabs; the pipeline counts from 0
  const int nchunks = (nkl + CHUNK_SLABS - 1) / CHUNK_SLABS;

  if (ep.chained) asm volatile("griddepcontrol.launch_dependents;");
  if (tid == NDRAIN_WARPS * 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapB) : "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, NDRAIN_WARPS * 32);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // the first product's slices come from the kernel before it
  if (!ep.chained) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
  }
  const uint32_t tmem = *tmem_slot;

  if (warp == NDRAIN_WARPS) {
    if (lane == 0) {
      // kind::f16: D F32 (bits 4-5 = 1), A BF16 (7-9 = 1), B BF16 (10-12 = 1), K-major both
      // instruction descriptor for an N-wide product (N = 64 .. 256, a multiple of 64 here)
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BM >> 4) << 24);
      auto idesc_n = [&](int n) { return idesc0 | ((uint32_t)(n >> 3) << 17); };
      auto a_ptr = [&](int st, int s) { return smem + st * STAGE_BYTES + s * SLICE_A; };
      auto b_ptr = [&](int st, int s) { return smem + st * STAGE_BYTES + S * SLICE_A + s * SLICE_B; };
      auto issue = [&](int t, int st) {
        mbar_expect_tx(&full[st], STAGE_BYTES);
        const int kc = (tb + t) * BKS;
        tma_load_3d(a_ptr(st, 0), &mapA, &full[st], kc, m0, (ep.a_batched ? bz : 0) * S);
        tma_load_3d(b_ptr(st, 0), &mapB, &full[st], kc, n0, (ep.b_batched ? bz : 0) * S);
      };
      const int pre = nkl < STAGES ? nkl : STAGES;
      for (int t = 0; t < pre; ++t) issue(t, t);
      int issued = pre;
      bool ok = true;
      for (int c = 0; c < nchunks && ok; ++c) {
        if (c >= 1 && !mbar_wait(accempty, (c - 1) & 1, fail)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int t0 = c * CHUNK_SLABS, t1 = min(nkl, t0 + CHUNK_SLABS);
        for (int t = t0; t < t1 && ok; ++t) {
          const int st = t % STAGES;
          if (!mbar_wait(&full[st], (t / STAGES) & 1, fail)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int kk = 0; kk < BKS / 16; ++kk) {
            const uint32_t off = kk * 32;  // 16 bf16 = 32 bytes inside the 64-byte swizzle atom
            // A^(s) meets B^(0..G-1-s) in one product of width (G-s) x BN: the B slices lie
            // back to back along N in shared memory (8-row groups 512 B apart throughout)
            // and the accumulators of groups s .. G-1 back to back in TMEM, so D columns
            // [s BN, G BN) += A^(s) [B^(0) | ... | B^(G-1-s)], split in widths <= 256.
            // (One 64-wide product per slice pair re-read A from shared memory 21 times.)
#pragma unroll
            for (int sa = 0; sa < S; ++sa) {
              const uint64_t ad = sdesc64(smem_u32(a_ptr(st, sa)) + off);
#pragma unroll
              for (int u0 = 0; u0 < G - sa; u0 += 4) {
                const int width = (G - sa - u0) >= 4 ? 4 * BN : (G - sa - u0) * BN;
                // every accumulator's first product of the chunk is the sa = 0 one at t0, kk 0
                mma_bf16(tmem + (uint32_t)((sa + u0) * BN), ad, sdesc64(smem_u32(b_ptr(st, u0)) + off),
                         idesc_n(width), (t == t0 && kk == 0 && sa == 0) ? 0u : 1u);
              }
            }
          }
          mma_commit(&empty[st]);
          if (t >= 1 && issued < nkl) {
            const int sp = (t - 1) % STAGES;
            if (!mbar_wait(&empty[sp], ((t - 1) / STAGES) & 1, fail)) {
              ok = false;
              break;
            }
            issue(issued, sp);
            ++issued;
          }
        }
        if (!ok) break;
        mma_commit(accfull);
      }
      if (!ok) {
        *fail = 1;
        atomicExch(ep.err, 1);
        for (int t = 0; t < issued; ++t) mbar_wait(&full[t % STAGES], (t / STAGES) & 1, nullptr);
      }
    }
  } else {
    // drain warps: warpgroup q = warp / 4 owns columns [16 q, 16 q + 16); TMEM lanes 32 (warp % 4) ..
    const int q = warp >> 2, wl = warp & 3;
    float hi[16], lo[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0.f;
    const uint32_t lane_base = (uint32_t)(wl * 32) << 16;
    // the scales' exponents, for the epilogue
    if (tid < BM)
      s_exp[tid] = pow2_exponent(ep.sa[(ep.a_batched ? bz : 0) * ep.Mp + m0 + tid]);
    else if (tid < BM + BN)
      s_exp[tid] = pow2_exponent(ep.sb[(ep.b_batched ? bz : 0) * ep.Np + n0 + tid - BM]);
    asm volatile("bar.sync 1, %0;" ::"n"(NDRAIN_WARPS * 32) : "memory");
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      if (!mbar_wait(accfull, c & 1, fail)) {
        ok = false;
        atomicExch(ep.err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // three groups' TMEM loads in flight per wait (one wait per group made the drain,
      // and with it the tensor pipe, wait on the load latency six times per chunk).  The
      // groups are added smallest first: the sums' low parts stay small, so their rounding
      // does too (K = 777, entries near one, eight slices: largest error 5.6e-12, against
      // 1.15e-11 largest first).  The last two groups go to the low part with one addition:
      // its rounding, 2^-24 of a term of 2^-7S, is below what the dropped groups are.
#pragma unroll
      for (int g0 = G - 1; g0 >= 0; g0 -= 3) {
        uint32_t r[3][16];
#pragma unroll
        for (int gg = 0; gg < 3; ++gg) {
          if (g0 - gg >= 0)
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                "%13, %14, %15}, [%16];"
                : "=r"(r[gg][0]), "=r"(r[gg][1]), "=r"(r[gg][2]), "=r"(r[gg][3]), "=r"(r[gg][4]), "=r"(r[gg][5]),
                  "=r"(r[gg][6]), "=r"(r[gg][7]), "=r"(r[gg][8]), "=r"(r[gg][9]), "=r"(r[gg][10]), "=r"(r[gg][11]),
                  "=r"(r[gg][12]), "=r"(r[gg][13]), "=r"(r[gg][14]), "=r"(r[gg][15])
                : "r"(tmem + lane_base + (uint32_t)((g0 - gg) * BN + 16 * q)));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (g0 < 3) {
          // the last loads are in registers: release the accumulators before the
          // arithmetic, so the next chunk's products overlap it
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          mbar_arrive(accempty);
        }
#pragma unroll
        for (int gg = 0; gg < 3; ++gg) {
          if (g0 - gg >= 0) {
            const float sc = __int_as_float((127 - 7 * (g0 - gg + 2)) << 23);  // 2^{-7(g+2)}, exact
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (g0 - gg >= G - 2)
                lo[j] = fmaf(__uint_as_float(r[gg][j]), sc, lo[j]);
              else
                two_sum_acc(hi[j], lo[j], __uint_as_float(r[gg][j]) * sc);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {  // renormalise (fast two-sum)
        float s = hi[j] + lo[j];
        lo[j] = lo[j] - (s - hi[j]);
        hi[j] = s;
      }
    }
    // a chained product updates C after the products before it, and ends after them; a partial
    // product is its own and need not wait to be written
    if (ep.nsplit == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (ok) {
      // Epilogue: no load between the stores (the scales' exponents are in shared memory) and
      // one FP64 operation per output (GB300 runs FP64 at ~2 per clock per SM) but for alpha and
      // beta: 6900 cycles a tile.  With the scales loaded between the stores, and conversions
      // and multiplications the compiler ran for every value, it took 34000 of the 46000 cycles
      // of a tile of depth 128 (integer arithmetic alone, correctly rounded: 9000).
      const int64_t row = m0 + wl * 32 + lane;
      const int ka = s_exp[wl * 32 + lane];
      double* Wz = ep.nsplit > 1 ? ep.W + (size_t)blockIdx.z * ep.M * ep.N : nullptr;
      const int ncol = int(min((int64_t)16, ep.N - (n0 + 16 * q)));
      if (row < ep.M && ncol > 0) {
        double* cp = Wz ? Wz + row + (n0 + 16 * q) * ep.M : ep.C + bz * ep.sC + row * ep.crs + (n0 + 16 * q) * ep.ldc;
        const int64_t step = Wz ? ep.M : ep.ldc;
#pragma unroll
        for (int h = 0; h < 16; h += 8) {
          double v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int kb = s_exp[BM + 16 * q + h + j];
            v[j] = join_pow2(hi[h + j], lo[h + j], ka + kb);
            if (ka > 1023 || kb > 1023) v[j] = __longlong_as_double(0x7ff8000000000000ll);  // a row that is not finite
          }
          if (!Wz && ep.alpha != 1.0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] *= ep.alpha;
          }
          if (!Wz && ep.beta != 0.0) {
            double old[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) old[j] = h + j < ncol ? cp[(h + j) * step] : 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = fma(ep.beta, old[j], v[j]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (h + j < ncol) cp[(h + j) * step] = v[j];
        }
      }
    }
    if (ep.nsplit > 1) asm volatile("griddepcontrol.wait;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// Products of one shape, C_t = alpha_t A_t B_t^T + beta_t C_t, in order (the parts of a complex
// product; two of them share a C)
struct OzTerms {
  int n;
  double* C[4];
  double alpha[4], beta[4];
};

// C_t = alpha_t sum_s W[t][b nsplit + s] + beta_t C_t for the terms from `first` on, the splits
// added in order
__global__ void oz_split_reduce_kernel(const double* W, int nsplit, int64_t M, int64_t N, int64_t batch,
                                       const __grid_constant__ OzTerms terms, int first, int64_t ldc, int64_t sC,
                                       int64_t crs) {
  chained_start();
  const int64_t MN = M * N, tot = MN * batch;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = e / MN, r = e - b * MN, row = r % M, col = r / M;
    for (int t = first; t < terms.n; ++t) {
      const double* Wt = W + (t - first) * nsplit * tot;
      double acc = 0.0;
      for (int sp = 0; sp < nsplit; ++sp) acc += Wt[(b * nsplit + sp) * MN + r];
      const double v = terms.alpha[t] == 1.0 ? acc : acc * terms.alpha[t];
      double* cp = terms.C[t] + b * sC + row * crs + col * ldc;
      *cp = (terms.beta[t] == 0.0) ? v : fma(terms.beta[t], *cp, v);
    }
  }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeFn)p;
  });
  return fn;
}

// slices [planes = batch*S][rows_p][K_p] bf16; box {32, box_rows, S}
CUtensorMap make_map(void* base, int64_t rows_p, int64_t K_p, int64_t planes, int box_rows, int S) {
  EncodeFn enc = encode_fn();
  NSG_CHECK(enc != nullptr, NSG_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  CUtensorMap m;
  cuuint64_t dims[3] = {(cuuint64_t)K_p, (cuuint64_t)rows_p, (cuuint64_t)planes};
  cuuint64_t strides[2] = {(cuuint64_t)(K_p * 2), (cuuint64_t)(K_p * rows_p * 2)};
  cuuint32_t box[3] = {(cuuint32_t)BKS, (cuuint32_t)box_rows, (cuuint32_t)S};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  NSG_CHECK(r == CUDA_SUCCESS, NSG_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return m;
}

// One operand of an Ozaki product, sliced: S bf16 slices [batch][S][rows_p][K_p] and the
// power-of-two row scales [batch][rows_p].
struct OzOperand {
  __nv_bfloat16* slices = nullptr;
  double* scales = nullptr;
  int64_t rows_p = 0, batch = 1;
};

// bytes of the slices, the scales and the slabs' row maxima (256-byte aligned each)
inline size_t oz_align(size_t b) { return (b + 255) & ~size_t(255); }
template <int S>
size_t oz_operand_bytes(int64_t rows_p, int64_t K_p, int64_t batch) {
  const size_t rows = size_t(rows_p) * batch;
  return oz_align(2 * size_t(S) * rows * K_p) + oz_align(8 * rows) +
         (K_p >= kShallow ? oz_align(4 * rows * ((K_p + kMaxSlab - 1) / kMaxSlab)) : 0);
}

// The operands of a product laid out in `mem`, one after the other, and sliced: op(X) viewed
// as rows x K (element (r, k) at src[b bs + r rs + k ks], in doubles).
template <int S>
struct OzSlicer {
  nsg_ctx* c;
  OzSources P{};
  unsigned char* mem;
  OzSlicer(nsg_ctx* cc, unsigned char* m, int64_t K, int64_t K_p) : c(cc), mem(m) {
    P.K = K;
    P.K_p = K_p;
  }
  OzOperand add(const double* src, int64_t rows, int64_t rs, int64_t ks, int64_t bs, int64_t batch, int64_t rows_p) {
    const size_t all = size_t(rows_p) * batch;
    OzOperand o;
    o.slices = (__nv_bfloat16*)mem;
    o.scales = (double*)(mem + oz_align(2 * size_t(S) * all * P.K_p));
    o.rows_p = rows_p;
    o.batch = batch;
    const int64_t before = P.n > 0 ? P.op[P.n - 1].tile_end : 0;
    P.op[P.n++] = OzSource{src, rows, rs, ks, bs, rows_p, batch, o.scales, (unsigned*)((char*)o.scales + oz_align(8 * all)),
                           o.slices, before + rows_p / kSliceRows * batch};
    mem += oz_operand_bytes<S>(rows_p, P.K_p, batch);
    return o;
  }
  void run() {
    ProfScope ps(c, NSG_PROF_SPLIT, 0.0);
    const int64_t tiles = P.op[P.n - 1].tile_end;
    if (P.K_p < kShallow && tiles * 8 < (1ll << 31)) {
      int C = 1;
      while (P.K_p > int64_t(kSliceK) * C) C *= 2;
      P.slab = int((P.K_p / 32 + C - 1) / C * 32);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(unsigned(tiles * C));
      cfg.blockDim = dim3(kSliceThreads);
      cfg.stream = c->stream;
      cudaLaunchAttribute attr[2] = {chained_attribute()};
      attr[1].id = cudaLaunchAttributeClusterDimension;
      attr[1].val.clusterDim.x = C;
      attr[1].val.clusterDim.y = 1;
      attr[1].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      NSG_CUDA(cudaLaunchKernelEx(&cfg, oz_slice_shallow_kernel<S>, P));
      count_launch(c);
    } else {
      const int slabs = int((P.K_p + kMaxSlab - 1) / kMaxSlab);
      NSG_CHECK(tiles < (1ll << 31), NSG_ERR_UNSUPPORTED, "ozaki slices: grid too large");
      // beyond 512 CTAs a row tile they take several slabs each: a CTA that slices reads the
      // maxima of all slabs, and a grid has 65535 rows (the loop costs the others 2 to 4 % of an
      // eigensolve at bond dimension 1024 and of an environment update)
      const int64_t yslice = (P.K_p + kSliceK - 1) / kSliceK;
      const bool many = yslice > 512;
      for (int o = 0; o < P.n; ++o) {
        const unsigned mine = unsigned(P.op[o].rows_p / kSliceRows * P.op[o].batch);
        if (many) {
          oz_row_max_kernel<true><<<dim3(mine, 512), kSliceThreads, 0, c->stream>>>(P.op[o], P.K, slabs);
          oz_slice_deep_kernel<S, true><<<dim3(mine, 512), kSliceThreads, 0, c->stream>>>(P.op[o], P.K, P.K_p, slabs);
        } else {
          oz_row_max_kernel<false><<<dim3(mine, slabs), kSliceThreads, 0, c->stream>>>(P.op[o], P.K, slabs);
          oz_slice_deep_kernel<S, false><<<dim3(mine, unsigned(yslice)), kSliceThreads, 0, c->stream>>>(P.op[o], P.K, P.K_p,
                                                                                                     slabs);
        }
      }
      count_launch(c, 2 * P.n);
    }
    check_launch("ozaki slices");
  }
};

// The terms' products of prepared operands (A[t], B[t]) into their C (stride ldc between
// columns, sC between batch entries, crs between rows; all in doubles).  The launches after
// the first are chained: they start while the one before still runs, on the SMs it leaves, and
// wait for it before their epilogue (a complex product with its slicing, 640 x 512 x 128, 40
// tiles a term: 104 us one term after the other, 77 chained; 4096 x 1024 x 1024: 909, 804).
template <int S>
void oz_products(nsg_ctx* c, const OzOperand* const* A, const OzOperand* const* B, const OzTerms& terms, int64_t M,
                 int64_t N, int64_t K_p, int64_t batch, int64_t ldc, int64_t sC, int64_t crs, int64_t flop_k) {
  constexpr int SMEM_BYTES = Oz<S>::SMEM_BYTES;
  const int64_t Mp = A[0]->rows_p, Np = B[0]->rows_p;
  int* err = device_flag(c);  // checked once at the end of the public call
  ensure_smem_limit((const void*)oz_gemm_kernel<S>, SMEM_BYTES);
  // split K when the output tiles would leave most SMs idle (the small products of a
  // converged sweep: 32-64 tiles of 128 x 64 on 152 SMs)
  const int nk = int(K_p / BKS), units = (nk + SPLIT_SLABS - 1) / SPLIT_SLABS;
  const int64_t tiles = (Mp / BM) * (Np / BN) * batch;
  const int64_t sms = c->num_sms > 0 ? c->num_sms : 152;
  int nsplit = 1;
  if (tiles * 2 <= sms && units >= 2)
    nsplit = int(std::min<int64_t>({(int64_t)units, sms / tiles, 16, 65535 / batch}));
  const int split_slabs = (units + nsplit - 1) / nsplit * SPLIT_SLABS;
  nsplit = (nk + split_slabs - 1) / split_slabs;
  // the partial products' workspace, only when K is split (freed on every exit): of all terms,
  // reduced together, or where that does not fit of one term at a time
  struct Partials {
    nsg_ctx* c;
    void* p;
    size_t bytes;
    ~Partials() {
      try {
        dfree(c, p, bytes);
      } catch (...) {
      }
    }
  } wbuf{c, nullptr, 0};
  const size_t term_w = size_t(nsplit) * size_t(batch) * size_t(M) * size_t(N);
  bool together = terms.n > 1;
  if (nsplit > 1) {
    for (;;) {
      const size_t bytes = sizeof(double) * term_w * (together ? terms.n : 1);
      try {
        wbuf.p = dalloc(c, bytes);
        wbuf.bytes = bytes;
        break;
      } catch (const Error& e) {
        if (!together || e.code != NSG_ERR_OOM) throw;
        together = false;
      }
    }
  }
  for (int t = 0; t < terms.n; ++t) {
    const CUtensorMap mA = make_map(A[t]->slices, Mp, K_p, S * A[t]->batch, BM, S),
                      mB = make_map(B[t]->slices, Np, K_p, S * B[t]->batch, BN, S);
    double* W = nsplit > 1 ? (double*)wbuf.p + (together ? t * term_w : 0) : nullptr;
    const OzEpi ep{terms.C[t],       ldc,          sC,           M,            N,   crs, terms.alpha[t], terms.beta[t],
                   A[t]->scales,     B[t]->scales, Mp,           Np,           A[t]->batch > 1, B[t]->batch > 1,
                   err,              nsplit,       split_slabs,  W,            t > 0 && (nsplit == 1 || together)};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(Mp / BM), unsigned(Np / BN), unsigned(batch * nsplit));
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1] = {chained_attribute()};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool reduce = nsplit > 1 && (!together || t + 1 == terms.n);
    ProfScope ps(c, NSG_PROF_TC_GEMM, 2.0 * double(M) * double(N) * double(flop_k) * double(batch));
    NSG_CUDA(cudaLaunchKernelEx(&cfg, oz_gemm_kernel<S>, mA, mB, nk, ep));
    if (reduce) {
      const int64_t tot = M * N * batch;
      const int rg = int(std::min<int64_t>((tot + 255) / 256, sms * 8));
      OzTerms upto = terms;
      upto.n = t + 1;
      launch_chained(c, oz_split_reduce_kernel, rg, 256, 0, (const double*)wbuf.p, nsplit, M, N, batch, upto,
                     together ? 0 : t, ldc, sC, crs);
    }
    count_launch(c, reduce ? 2 : 1);
  }
  check_launch("oz_gemm");
}

template <int S>
bool gemm_ozaki_impl(nsg_ctx* c, const GemmArgs& g) {
  if (g.dtype != NSG_F64 && g.dtype != NSG_C128) return false;
  if (!tensor_core_sizes(NSG_PREC_OZAKI, double(g.M), double(g.N), double(g.K))) return false;
  if (g.batch > 65535) return false;
  const bool cplx = g.dtype == NSG_C128;
  if (!cplx && (g.opA == OP_C || g.opA == OP_R || g.opB == OP_C || g.opB == OP_R)) return false;
  // complex: real scalars only (the four real products carry the signs)
  if (cplx && (g.alpha_im != 0.0 || g.beta_im != 0.0)) return false;
  const int64_t Mp = (g.M + BM - 1) / BM * BM, Np = (g.N + BN - 1) / BN * BN, Kp = (g.K + BKS - 1) / BKS * BKS;
  const bool transA = g.opA == OP_T || g.opA == OP_C, transB = g.opB == OP_T || g.opB == OP_C;
  const int64_t ars = !transA ? 1 : g.lda, aks = !transA ? g.lda : 1;
  const int64_t brs = !transB ? g.ldb : 1, bks = !transB ? 1 : g.ldb;
  const int64_t ab = (g.strideA == 0) ? 1 : g.batch, bb = (g.strideB == 0) ? 1 : g.batch;
  const size_t opA_bytes = oz_operand_bytes<S>(Mp, Kp, ab), opB_bytes = oz_operand_bytes<S>(Np, Kp, bb);
  if (!cplx) {
    ScopedBuf sbuf(c, opA_bytes + opB_bytes);
    unsigned char* buf = (unsigned char*)sbuf.p;
    OzSlicer<S> sl(c, buf, g.K, Kp);
    OzOperand A = sl.add((const double*)g.A, g.M, ars, aks, g.strideA, ab, Mp);
    OzOperand B = sl.add((const double*)g.B, g.N, brs, bks, g.strideB, bb, Np);
    sl.run();
    const OzOperand *pa[1] = {&A}, *pb[1] = {&B};
    const OzTerms terms{1, {(double*)g.C}, {g.alpha_re}, {g.beta_re}};
    oz_products<S>(c, pa, pb, terms, g.M, g.N, Kp, g.batch, g.ldc, g.strideC, 1, g.K);
    return true;
  }
  // complex: A = Ar + i sa Ai, B = Br + i sb Bi (sa, sb = -1 for conjugated operands), as
  // four real products on the interleaved parts (strides doubled, imaginary parts at +1):
  //   Re C = alpha (Ar Br - sa sb Ai Bi) + beta Re C,  Im C = alpha (sb Ar Bi + sa Ai Br) + beta Im C
  const double sa = (g.opA == OP_C || g.opA == OP_R) ? -1.0 : 1.0;
  const double sbs = (g.opB == OP_C || g.opB == OP_R) ? -1.0 : 1.0;
  ScopedBuf sbuf(c, 2 * (opA_bytes + opB_bytes));
  unsigned char* buf = (unsigned char*)sbuf.p;
  const double* Ad = (const double*)g.A;
  const double* Bd = (const double*)g.B;
  OzSlicer<S> sl(c, buf, g.K, Kp);
  OzOperand Ar = sl.add(Ad, g.M, 2 * ars, 2 * aks, 2 * g.strideA, ab, Mp);
  OzOperand Ai = sl.add(Ad + 1, g.M, 2 * ars, 2 * aks, 2 * g.strideA, ab, Mp);
  OzOperand Br = sl.add(Bd, g.N, 2 * brs, 2 * bks, 2 * g.strideB, bb, Np);
  OzOperand Bi = sl.add(Bd + 1, g.N, 2 * brs, 2 * bks, 2 * g.strideB, bb, Np);
  sl.run();
  double* Cr = (double*)g.C;
  const double al = g.alpha_re, be = g.beta_re;
  const OzOperand *pa[4] = {&Ar, &Ai, &Ar, &Ai}, *pb[4] = {&Br, &Bi, &Bi, &Br};
  const OzTerms terms{4, {Cr, Cr, Cr + 1, Cr + 1}, {al, -sa * sbs * al, sbs * al, sa * al}, {be, 1.0, be, 1.0}};
  oz_products<S>(c, pa, pb, terms, g.M, g.N, Kp, g.batch, 2 * g.ldc, 2 * g.strideC, 2, g.K);
  return true;
}

}  // namespace

bool gemm_ozaki_tc(nsg_ctx* c, const GemmArgs& g, int slices) {
  if (slices == 8) return gemm_ozaki_impl<8>(c, g);
  return gemm_ozaki_impl<6>(c, g);
}

}  // namespace nsg
