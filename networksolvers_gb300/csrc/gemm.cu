// FP64 / complex-FP64 strided-batched GEMM on the CUDA cores (the plain form).
//
// C_b = alpha * op(A_b) * op(B_b) + beta * C_b, column-major, op in {N, T, C, R}.
// GB300 executes FP64 at a small fraction of its FP32 rate, so this kernel is
// compute-bound for every shape that matters: 64x64 tiles with 4x4 outputs per thread for
// outputs that fill whole waves of SMs, 16x16 tiles with a cluster split of K for all
// others, and a row-per-thread form for products with a sparse operator tensor.  Loads
// are mapped so that consecutive threads touch consecutive addresses for either operand
// orientation.
#include "chained.h"
#include "nsg_internal.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

namespace nsg {

namespace {

constexpr int BM = 64, BN = 64, NT = 256;

__device__ __forceinline__ double ld(const double* p, bool) { return *p; }
__device__ __forceinline__ double2 ld(const double2* p, bool conj) {
  double2 v = *p;
  if (conj) v.y = -v.y;
  return v;
}
__device__ __forceinline__ void zero(double& v) { v = 0.0; }
__device__ __forceinline__ bool nonzero(double v) { return v != 0.0; }
__device__ __forceinline__ bool nonzero(double2 v) { return v.x != 0.0 || v.y != 0.0; }
__device__ __forceinline__ void zero(double2& v) { v = make_double2(0.0, 0.0); }
__device__ __forceinline__ double plus(double a, double b) { return a + b; }
__device__ __forceinline__ double2 plus(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ void mac(double& acc, double a, double b) { acc = fma(a, b, acc); }
__device__ __forceinline__ void mac(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}

// shift of a coefficient +-2^s with |s| < 512 as 2 s + (negative), `none` for any other
// value; and a times that coefficient: by adding s to a's exponent field and flipping its
// sign bit when the result is a normal number, else by the multiplication (same value)
__device__ __forceinline__ int pow2_shift(double v, int none) {
  const long long b = __double_as_longlong(v);
  const int s = int((b >> 52) & 0x7ff) - 1023;
  if ((b & 0xfffffffffffffll) != 0 || s <= -512 || s >= 512) return none;
  return 2 * s + (b < 0 ? 1 : 0);
}
__device__ __forceinline__ int pow2_shift(double2 v, int none) { return v.y == 0.0 ? pow2_shift(v.x, none) : none; }
__device__ __forceinline__ double mul_pow2(double a, int code, double v) {
  const long long b = __double_as_longlong(a);
  const int e = int((b >> 52) & 0x7ff), s = code >> 1;
  if (e == 0x7ff || e == 0 || e + s <= 0 || e + s >= 0x7ff) return a * v;
  return __longlong_as_double((b + ((long long)s << 52)) ^ ((long long)(code & 1) << 63));
}
__device__ __forceinline__ double2 mul_pow2(double2 a, int code, double2 v) {
  return make_double2(mul_pow2(a.x, code, v.x), mul_pow2(a.y, code, v.x));
}

template <typename T>
struct Scal;
template <>
struct Scal<double> {
  double a, b;
  __device__ double epi(double acc, const double* c) const { return b == 0.0 ? a * acc : fma(a, acc, b * (*c)); }
};
template <>
struct Scal<double2> {
  double2 a, b;
  __device__ double2 epi(double2 acc, const double2* c) const {
    double2 r = make_double2(a.x * acc.x - a.y * acc.y, a.x * acc.y + a.y * acc.x);
    if (b.x != 0.0 || b.y != 0.0) {
      double2 cv = *c;
      r.x += b.x * cv.x - b.y * cv.y;
      r.y += b.x * cv.y + b.y * cv.x;
    }
    return r;
  }
};

// splits > 1: grid z covers batch * splits; split sp sums k in [sp*ksplit, (sp+1)*ksplit)
// and writes its raw partial product to C + bz * M * N (ld = M); a reduction applies
// alpha / beta afterwards in a fixed order.
template <typename T, int BK>
__global__ void __launch_bounds__(NT)
    gemm_kernel(int64_t M, int64_t N, int64_t Kfull, const T* __restrict__ A, int64_t lda, int64_t sA, int opA,
                const T* __restrict__ B, int64_t ldb, int64_t sB, int opB, T* __restrict__ C, int64_t ldc,
                int64_t sC, int64_t batch, Scal<T> sc, int splits, int64_t ksplit) {
  __shared__ T As[BK][BM + 1];
  __shared__ T Bs[BK][BN + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t m0 = int64_t(blockIdx.x) * BM, n0 = int64_t(blockIdx.y) * BN;
  const bool transA = (opA == OP_T || opA == OP_C), conjA = (opA == OP_C || opA == OP_R);
  const bool transB = (opB == OP_T || opB == OP_C), conjB = (opB == OP_C || opB == OP_R);
  for (int64_t bzz = blockIdx.z; bzz < batch * splits; bzz += gridDim.z) {
    const int64_t bz = bzz / splits, sp = bzz % splits;
    const int64_t kb = sp * ksplit;
    const int64_t K = (splits > 1) ? ((kb + ksplit < Kfull) ? ksplit : Kfull - kb) : Kfull;
    const T* Ab = A + bz * sA + (transA ? kb : kb * lda);
    const T* Bb = B + bz * sB + (transB ? kb * ldb : kb);
    T* Cb = (splits > 1) ? C + bzz * M * N : C + bz * sC;
    const int64_t ldcc = (splits > 1) ? M : ldc;
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) zero(acc[i][j]);
    for (int64_t k0 = 0; k0 < K; k0 += BK) {
      // A tile: BM x BK
#pragma unroll
      for (int r = 0; r < (BM * BK) / NT; ++r) {
        int e = threadIdx.x + r * NT;
        int i, k;
        if (!transA) {
          i = e % BM;
          k = e / BM;
        } else {
          k = e % BK;
          i = e / BK;
        }
        int64_t gi = m0 + i, gk = k0 + k;
        T v;
        zero(v);
        if (gi < M && gk < K) v = ld(transA ? Ab + gk + gi * lda : Ab + gi + gk * lda, conjA);
        As[k][i] = v;
      }
      // B tile: BK x BN
#pragma unroll
      for (int r = 0; r < (BN * BK) / NT; ++r) {
        int e = threadIdx.x + r * NT;
        int j, k;
        if (!transB) {
          k = e % BK;
          j = e / BK;
        } else {
          j = e % BN;
          k = e / BN;
        }
        int64_t gj = n0 + j, gk = k0 + k;
        T v;
        zero(v);
        if (gj < N && gk < K) v = ld(transB ? Bb + gj + gk * ldb : Bb + gk + gj * ldb, conjB);
        Bs[k][j] = v;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        T a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = As[k][ty + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) mac(acc[i][j], a[i], b[j]);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int64_t gi = m0 + ty + 16 * i;
      if (gi >= M) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int64_t gj = n0 + tx + 16 * j;
        if (gj >= N) continue;
        T* cp = Cb + gi + gj * ldcc;
        if (splits > 1)
          *cp = acc[i][j];
        else
          *cp = sc.epi(acc[i][j], cp);
      }
    }
  }
}

template <typename T>
__global__ void splitk_reduce_kernel(int64_t M, int64_t N, int64_t batch, int splits, const T* __restrict__ W,
                                     T* __restrict__ C, int64_t ldc, int64_t sC, Scal<T> sc) {
  const int64_t MN = M * N, tot = MN * batch;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < tot; e += int64_t(gridDim.x) * blockDim.x) {
    int64_t b = e / MN, r = e % MN, i = r % M, j = r / M;
    T acc;
    zero(acc);
    for (int sp = 0; sp < splits; ++sp) {
      T v = W[(b * splits + sp) * MN + r];
      if constexpr (sizeof(T) == 8) {
        acc += v;
      } else {
        acc.x += v.x;
        acc.y += v.y;
      }
    }
    T* cp = C + b * sC + i + j * ldc;
    *cp = sc.epi(acc, cp);
  }
}

// Small-tile form: one 16 x 16 output tile per CTA of 256 threads (one output each), K cut
// into `splits` slices held by the CTAs of one thread-block cluster.  An SM retires two
// FP64 multiply-adds per clock and a warp's one holds its sub-partition's pipe for 64
// clocks, so neither register blocking nor operand traffic matters (a tile's operands are
// re-read from L2 at 1 byte per multiply-add): small tiles waste the least work on padding
// and fill the SMs evenly.  Measured against 32 x 32 tiles (2 x 2 to 2 x 4 outputs per
// thread) and 16 x 16 tiles of 128 threads or with K dealt to the warps: fastest or within
// 2 % at every size from 36^2 to 2072 x 924.  The slices' partial tiles are added through
// distributed shared memory in rank order: no workspace, no second launch.  The next K slab
// is loaded into registers while the current one is multiplied.  With launch, 64^3: 8 us
// (64 x 64 tiles with split K: 29), 128^3: 12 (31), 256^3: 41 (49), 2072 x 924 x 259: 0.85 ms
// (1.10); complex 64^3: 12 (77), 512^3: 0.95 ms (1.06).
constexpr int TB = 16, kTileThreads = TB * TB;
template <typename T, int BK>
__global__ void __launch_bounds__(kTileThreads)
    gemm_tile_kernel(int64_t M, int64_t N, int64_t Kfull, const T* __restrict__ A, int64_t lda, int64_t sA, int opA,
                     const T* __restrict__ B, int64_t ldb, int64_t sB, int opB, T* __restrict__ C, int64_t ldc,
                     int64_t sC, int64_t batch, Scal<T> sc, int splits, int64_t kslice) {
  constexpr int NL = BK / TB;
  __shared__ T As[2][BK][TB + 1], Bs[2][BK][TB + 1];
  __shared__ T Cs[kTileThreads];
  const int tid = threadIdx.x, ti = tid % TB, tj = tid / TB;
  const int64_t m0 = int64_t(blockIdx.x) * TB, n0 = int64_t(blockIdx.y) * TB;
  const bool transA = (opA == OP_T || opA == OP_C), conjA = (opA == OP_C || opA == OP_R);
  const bool transB = (opB == OP_T || opB == OP_C), conjB = (opB == OP_C || opB == OP_R);
  const int64_t zstep = int64_t(gridDim.z) / splits;  // splits > 1: grid z is exactly batch x splits
  const int sp = int(blockIdx.z % unsigned(splits));
  const int64_t kb = sp * kslice, K = max(int64_t(0), min(kslice, Kfull - kb));
  for (int64_t bz = blockIdx.z / unsigned(splits); bz < batch; bz += zstep) {
    const T* Ab = A + bz * sA;
    const T* Bb = B + bz * sB;
    T ra[NL], rb[NL];
    // lanes run along the contiguous axis of each operand as stored
    auto load = [&](int64_t k0) {
#pragma unroll
      for (int r = 0; r < NL; ++r) {
        const int i = transA ? tj : ti, ka = (transA ? ti : tj) + TB * r;
        const int j = transB ? ti : tj, kc = (transB ? tj : ti) + TB * r;
        const int64_t gi = m0 + i, gka = kb + k0 + ka, gj = n0 + j, gkb = kb + k0 + kc;
        zero(ra[r]);
        zero(rb[r]);
        if (gi < M && k0 + ka < K) ra[r] = ld(transA ? Ab + gka + gi * lda : Ab + gi + gka * lda, conjA);
        if (gj < N && k0 + kc < K) rb[r] = ld(transB ? Bb + gj + gkb * ldb : Bb + gkb + gj * ldb, conjB);
      }
    };
    T acc;
    zero(acc);
    load(0);
    int buf = 0;
    for (int64_t k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
#pragma unroll
      for (int r = 0; r < NL; ++r) {
        As[buf][(transA ? ti : tj) + TB * r][transA ? tj : ti] = ra[r];
        Bs[buf][(transB ? tj : ti) + TB * r][transB ? ti : tj] = rb[r];
      }
      __syncthreads();  // (the other buffer's readers passed the previous slab's barrier)
      if (k0 + BK < K) load(k0 + BK);
      const int kn = int(min(int64_t(BK), K - k0));
      if (kn == BK) {
#pragma unroll
        for (int k = 0; k < BK; ++k) mac(acc, As[buf][k][ti], Bs[buf][k][tj]);
      } else {  // the ragged last slab: no multiply-adds on its padding
        for (int k = 0; k < kn; ++k) mac(acc, As[buf][k][ti], Bs[buf][k][tj]);
      }
    }
    T* Cb = C + bz * sC;
    if (splits == 1) {
      const int64_t gi = m0 + ti, gj = n0 + tj;
      if (gi < M && gj < N) {
        T* cp = Cb + gi + gj * ldc;
        *cp = sc.epi(acc, cp);
      }
      __syncthreads();  // this batch entry's slabs are read before the next one's are stored
    } else {
      namespace cg = cooperative_groups;
      cg::cluster_group cluster = cg::this_cluster();
      Cs[tid] = acc;
      cluster.sync();
      const int per = kTileThreads / splits, e = sp * per + tid;
      const int64_t gi = m0 + e % TB, gj = n0 + e / TB;
      if (tid < per && gi < M && gj < N) {
        T sum = *cluster.map_shared_rank(Cs + e, 0);
        for (int r = 1; r < splits; ++r) sum = plus(sum, *cluster.map_shared_rank(Cs + e, r));
        T* cp = Cb + gi + gj * ldc;
        *cp = sc.epi(sum, cp);
      }
      cluster.sync();  // no CTA leaves while another may still read its tile
    }
  }
}

// Tall-skinny products with N, K <= 32: the site-operator steps of H_eff and of the
// environment updates (K, N = w d, batched over the other bond).  op(B) is an MPO tensor
// and mostly zeros: each CTA stages it in shared memory and lists the non-zeros of every
// column (one warp per column, ballots), and a warp forms 32 rows of its columns of C from
// exactly their non-zeros, on a [k][row] tile of op(A).  A column's multiply-adds are a
// chain of 64 clocks each, so with few rows the columns are dealt to up to CW = 8 warps
// and with many to one.  The rows of all batch entries that share B (strideB = 0) form one
// row space, so short batch entries fill whole CTAs.  The FP64 pipe (two multiply-adds per
// clock and SM) bounds the kernel beside the HBM traffic of A and C, so a column's first
// term is an exponent addition where its coefficient is a power of two (half of an MPO's
// entries) and alpha = 1, beta = 0 cost nothing.  216 rows, N = K = 18 complex: 20 us with
// one warp listing B and a row per thread, 15 with the parallel list, 6 with the columns
// dealt out.
constexpr int kSkinnyThreads = 256;
template <typename T, int CW>
__global__ void __launch_bounds__(kSkinnyThreads)
    gemm_skinny_kernel(int64_t M, int64_t rows, int N, int K, const T* __restrict__ A_, int64_t lda, int64_t sA,
                       bool conjA, const T* __restrict__ B_, int64_t ldb, int64_t sB, int opB, T* __restrict__ C,
                       int64_t ldc, int64_t sC, int64_t groups, Scal<T> sc, bool plain) {
  extern __shared__ __align__(16) unsigned char sk_smem[];
  // (many rows, CW = 1: not chained, and the loads through the read-only path)
  if constexpr (CW > 1) chained_start();
  const T* __restrict__ A = CW > 1 ? after_start(A_) : A_;
  const T* __restrict__ B = CW > 1 ? after_start(B_) : B_;
  constexpr int R = kSkinnyThreads / CW;     // rows per CTA
  T* As = (T*)sk_smem;                       // [K][R]
  __shared__ T Bs[32][33];                   // op(B)
  __shared__ T nzv[32][32];                  // non-zeros of each column of op(B)
  __shared__ unsigned char nzk[32][32];      // their row index k
  __shared__ int cnt[32], lead[32];          // their number; exponent of a real power-of-two first one
  constexpr int kNoLead = 1 << 20;
  const bool transB = (opB == OP_T || opB == OP_C), conjB = (opB == OP_C || opB == OP_R);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = kSkinnyThreads / 32;
  const int rl = tid % R, cw = tid / R;  // row in the tile, first column
  const int64_t tiles = (rows + R - 1) / R;
  int64_t listed = -1;
  for (int64_t job = blockIdx.x; job < tiles * groups; job += gridDim.x) {
    const int64_t g = job / tiles, r = (job % tiles) * R + rl;
    const int64_t bz = g + r / M, i = r % M;  // (groups > 1: rows = M, so r / M = 0)
    __syncthreads();  // the previous job's readers are done
    if (g != listed) {
      const T* Bb = B + g * sB;
      for (int e = tid; e < N * K; e += kSkinnyThreads) {
        const int j = transB ? e % N : e / K, k = transB ? e / N : e % K;
        Bs[j][k] = ld(transB ? Bb + j + (int64_t)k * ldb : Bb + k + (int64_t)j * ldb, conjB);
      }
    }
    T* Ar = As + rl;
    if (r < rows) {
      const T* Ab = A + bz * sA + i;
#pragma unroll 8
      for (int k = cw; k < K; k += CW) Ar[k * R] = ld(Ab + (int64_t)k * lda, conjA);
    }
    __syncthreads();
    if (g != listed) {
      for (int j = warp; j < N; j += nw) {
        T v;
        zero(v);
        if (lane < K) v = Bs[j][lane];
        const unsigned m = __ballot_sync(0xffffffffu, nonzero(v));
        if (nonzero(v)) {
          const int pos = __popc(m & ((1u << lane) - 1u));
          nzv[j][pos] = v;
          nzk[j][pos] = (unsigned char)lane;
          if (pos == 0) lead[j] = pow2_shift(v, kNoLead);
        }
        if (lane == 0) cnt[j] = __popc(m);
      }
      listed = g;
      __syncthreads();
    }
    if (r < rows) {
      T* Cb = C + bz * sC + i;
      for (int j = cw; j < N; j += CW) {
        const int c = cnt[j];
        T acc;
        zero(acc);
        int t = 0;
        if (c > 0) {
          const T a = Ar[nzk[j][0] * R];
          if (lead[j] != kNoLead)
            acc = mul_pow2(a, lead[j], nzv[j][0]);
          else
            mac(acc, a, nzv[j][0]);
          t = 1;
        }
        for (; t < c; ++t) mac(acc, Ar[nzk[j][t] * R], nzv[j][t]);
        T* cp = Cb + (int64_t)j * ldc;
        *cp = plain ? acc : sc.epi(acc, cp);
      }
    }
  }
}

template <typename T, int BK>
void launch_tile(nsg_ctx* c, const GemmArgs& g, Scal<T> sc, int splits, int64_t kslice) {
  cudaLaunchConfig_t cfg = {};
  const int64_t z = std::min<int64_t>(g.batch * splits, 65535);
  cfg.gridDim = dim3(unsigned((g.M + TB - 1) / TB), unsigned((g.N + TB - 1) / TB), unsigned(z));
  cfg.blockDim = dim3(kTileThreads);
  cfg.stream = c->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = unsigned(splits);
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  NSG_CUDA(cudaLaunchKernelEx(&cfg, gemm_tile_kernel<T, BK>, g.M, g.N, g.K, (const T*)g.A, g.lda, g.strideA, g.opA,
                              (const T*)g.B, g.ldb, g.strideB, g.opB, (T*)g.C, g.ldc, g.strideC, g.batch, sc, splits,
                              kslice));
}

// The 16 x 16 tiles unless the 64 x 64 tiles fill whole waves of SMs: both run the FP64
// pipe at its rate (96 % and 98 % of two multiply-adds per clock and SM measured on large
// products), so the line is where the last wave's idle SMs and the padding cost less than
// that difference.  K is split only while the tiles leave half of the SMs idle, into slices
// of at least 16 (more CTAs than SMs lose to the slices' fixed cost: 256^3 takes 42 us
// whole, 51 us in two slices).
bool gemm_small_tiles(nsg_ctx* c, const GemmArgs& g, int64_t sms, double flops) {
  auto tiles = [&](int64_t t) { return ((g.M + t - 1) / t) * ((g.N + t - 1) / t) * g.batch; };
  if (g.K < 1 || (g.N + TB - 1) / TB > 65535 || (g.M + TB - 1) / TB >= (1ll << 31)) return false;
  if (double((tiles(BM) + sms - 1) / sms * sms) * BM * BN < double(tiles(TB)) * TB * TB * 1.02) return false;
  int splits = 1;
  while (splits < 8 && tiles(TB) * splits * 2 <= sms && g.K >= 32 * splits) splits *= 2;
  const int64_t kslice = splits == 1 ? g.K : ((g.K + splits - 1) / splits + 3) / 4 * 4;
  ProfScope ps(c, NSG_PROF_SIMT_GEMM, flops);
  if (g.dtype == NSG_C128)
    launch_tile<double2, 16>(
        c, g, Scal<double2>{make_double2(g.alpha_re, g.alpha_im), make_double2(g.beta_re, g.beta_im)}, splits, kslice);
  else
    launch_tile<double, 32>(c, g, Scal<double>{g.alpha_re, g.beta_re}, splits, kslice);
  count_launch(c);
  check_launch("gemm_tile");
  return true;
}

}  // namespace

void gemm_f64_simt(nsg_ctx* c, const GemmArgs& g) {
  if (g.M == 0 || g.N == 0 || g.batch == 0) return;
  const int64_t sms = c->num_sms > 0 ? c->num_sms : 152;
  const bool cplx = g.dtype == NSG_C128;
  const double flops = double(g.M) * double(g.N) * double(g.K) * double(g.batch) * (cplx ? 8.0 : 2.0);
  if (g.N <= 32 && g.K <= 32 && g.K >= 1 && (g.opA == OP_N || g.opA == OP_R)) {
    // batch entries that share B are one row space; the columns on as many warps as it
    // takes to give each SM sub-partition a warp or two (32 rows each)
    const bool shared_b = g.strideB == 0 || g.batch == 1;
    const int64_t groups = shared_b ? 1 : g.batch, rows = shared_b ? g.M * g.batch : g.M;
    int col_warps = 1;
    while (col_warps < 8 && (rows + 31) / 32 * groups * col_warps < 8 * sms) col_warps *= 2;
    const bool plain = g.alpha_re == 1.0 && g.alpha_im == 0.0 && g.beta_re == 0.0 && g.beta_im == 0.0;
    ProfScope ps(c, NSG_PROF_SIMT_GEMM, flops);
    auto launch = [&](auto cw, auto sc) {
      using T = std::remove_reference_t<decltype(sc.a)>;
      constexpr int CW = decltype(cw)::value, R = kSkinnyThreads / CW;
      const int grid = int(std::min<int64_t>((rows + R - 1) / R * groups, sms * 16));
      ensure_smem_limit((const void*)gemm_skinny_kernel<T, CW>, 32 * R * int(sizeof(T)));
      const auto launch = [&](auto... args) {
        const size_t smem = size_t(g.K) * R * sizeof(T);
        if constexpr (CW > 1)
          launch_chained(c, gemm_skinny_kernel<T, CW>, grid, kSkinnyThreads, smem, args...);
        else
          gemm_skinny_kernel<T, CW><<<grid, kSkinnyThreads, smem, c->stream>>>(args...);
      };
      launch(g.M, rows, int(g.N), int(g.K), (const T*)g.A, g.lda, g.strideA, g.opA == OP_R, (const T*)g.B, g.ldb,
             g.strideB, g.opB, (T*)g.C, g.ldc, g.strideC, groups, sc, plain);
    };
    auto pick = [&](auto sc) {
      if (col_warps == 1)
        launch(std::integral_constant<int, 1>{}, sc);
      else if (col_warps == 2)
        launch(std::integral_constant<int, 2>{}, sc);
      else if (col_warps == 4)
        launch(std::integral_constant<int, 4>{}, sc);
      else
        launch(std::integral_constant<int, 8>{}, sc);
    };
    if (cplx)
      pick(Scal<double2>{make_double2(g.alpha_re, g.alpha_im), make_double2(g.beta_re, g.beta_im)});
    else
      pick(Scal<double>{g.alpha_re, g.beta_re});
    count_launch(c);
    check_launch("gemm_skinny");
    return;
  }
  if (c->tune_splitk == 0 && gemm_small_tiles(c, g, sms, flops)) return;
  int64_t gx = (g.M + BM - 1) / BM, gy = (g.N + BN - 1) / BN;
  NSG_CHECK(gx < (1ll << 31) && gy < 65536, NSG_ERR_UNSUPPORTED, "gemm: grid too large");
  // K is split here only by the context's override: without one, products of few tiles
  // are the small tiles' (above), which split K themselves
  int splits = 1;
  int64_t ksplit = g.K;
  if (c->tune_splitk > 0) {
    splits = int(std::min<int64_t>(c->tune_splitk, std::max<int64_t>(1, g.K / 16)));
    ksplit = (g.K + splits - 1) / splits;
    ksplit = ((ksplit + 15) / 16) * 16;
    splits = int((g.K + ksplit - 1) / ksplit);
  }
  int64_t zt = g.batch * splits;
  int64_t gz = zt < 65535 ? zt : 65535;
  dim3 grid{unsigned(gx), unsigned(gy), unsigned(gz)};
  const size_t eb = cplx ? 16 : 8;
  ProfScope ps(c, NSG_PROF_SIMT_GEMM, flops);
  void* W = nullptr;
  size_t wbytes = 0;
  void* Cout = g.C;
  if (splits > 1) {
    wbytes = eb * size_t(g.M) * size_t(g.N) * size_t(zt);
    W = dalloc(c, wbytes);
    Cout = W;
  }
  if (cplx) {
    Scal<double2> sc{make_double2(g.alpha_re, g.alpha_im), make_double2(g.beta_re, g.beta_im)};
    gemm_kernel<double2, 8><<<grid, NT, 0, c->stream>>>(g.M, g.N, g.K, (const double2*)g.A, g.lda, g.strideA, g.opA,
                                                        (const double2*)g.B, g.ldb, g.strideB, g.opB,
                                                        (double2*)Cout, g.ldc, g.strideC, g.batch, sc, splits, ksplit);
    if (splits > 1) {
      int64_t tot = g.M * g.N * g.batch;
      int rb = int(std::min<int64_t>((tot + 255) / 256, sms * 8));
      splitk_reduce_kernel<double2><<<rb, 256, 0, c->stream>>>(g.M, g.N, g.batch, splits, (const double2*)W,
                                                              (double2*)g.C, g.ldc, g.strideC, sc);
      count_launch(c);
    }
  } else {
    Scal<double> sc{g.alpha_re, g.beta_re};
    gemm_kernel<double, 16><<<grid, NT, 0, c->stream>>>(g.M, g.N, g.K, (const double*)g.A, g.lda, g.strideA, g.opA,
                                                        (const double*)g.B, g.ldb, g.strideB, g.opB, (double*)Cout,
                                                        g.ldc, g.strideC, g.batch, sc, splits, ksplit);
    if (splits > 1) {
      int64_t tot = g.M * g.N * g.batch;
      int rb = int(std::min<int64_t>((tot + 255) / 256, sms * 8));
      splitk_reduce_kernel<double><<<rb, 256, 0, c->stream>>>(g.M, g.N, g.batch, splits, (const double*)W,
                                                             (double*)g.C, g.ldc, g.strideC, sc);
      count_launch(c);
    }
  }
  if (W) dfree(c, W, wbytes);
  count_launch(c);
  check_launch("gemm_f64_simt");
}

// FP64-level products: the eight-slice Ozaki tensor-core form (within 4 K 2^-48 of the row and
// column scales' product, the bound of its FP32 accumulator pair) when the split precision is
// selected, otherwise the FP64 CUDA cores (never TF32x3).
void gemm_accurate(nsg_ctx* c, const GemmArgs& g_in) {
  GemmArgs g = g_in;
  if (g.dtype == NSG_F64) {
    if (g.opA == OP_C) g.opA = OP_T;
    if (g.opA == OP_R) g.opA = OP_N;
    if (g.opB == OP_C) g.opB = OP_T;
    if (g.opB == OP_R) g.opB = OP_N;
  }
  if ((c->precision == NSG_PREC_OZAKI || c->precision == NSG_PREC_OZAKI8) && gemm_ozaki_tc(c, g, 8)) return;
  gemm_f64_simt(c, g);
}

void gemm(nsg_ctx* c, const GemmArgs& g_in) {
  GemmArgs g = g_in;
  if (g.dtype == NSG_F64) {  // conjugation is the identity on real data
    if (g.opA == OP_C) g.opA = OP_T;
    if (g.opA == OP_R) g.opA = OP_N;
    if (g.opB == OP_C) g.opB = OP_T;
    if (g.opB == OP_R) g.opB = OP_N;
  }
  double mac = double(g.M) * double(g.N) * double(g.K) * double(g.batch);
  c->flops += uint64_t(mac * (g.dtype == NSG_C128 ? 8.0 : 2.0));
  if (g.K == 0) {
    // C = beta*C (alpha term vanishes)
    return;
  }
  if (c->precision == NSG_PREC_TF32X3 && gemm_split_tc(c, g)) return;
  if (c->precision == NSG_PREC_OZAKI && gemm_ozaki_tc(c, g, 6)) return;
  if (c->precision == NSG_PREC_OZAKI8 && gemm_ozaki_tc(c, g, 8)) return;
  gemm_f64_simt(c, g);
}

}  // namespace nsg
