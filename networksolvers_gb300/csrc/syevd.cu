// Dense Hermitian eigensolver for the truncated factorizations:
//   1. Householder reduction to a real symmetric tridiagonal T with the matrix in shared
//      memory, of one thread-block cluster (orders up to the tuning table's limit) or of
//      all SMs (real orders to ~1770, complex ~1210); beyond that one cooperative kernel
//      with one grid barrier per column (the matrix stays L2-resident),
//   2. Cuppen divide and conquer on T (dc.cu),
//   3. back-transformation of the kept eigenvectors with the Householder reflectors
//      in blocks of 64 (compact WY, three GEMMs per block; every block's T factor is
//      formed up front in one launch).
// The merge GEMMs and the two large back-transformation GEMMs use the FP64-level
// products (eight-slice Ozaki form in the split precision); the reflector Gram matrix
// V^H V and T W stay on the FP64 cores (six-slice products there alone cost 1e-11 of
// orthogonality).
// Every wait in these kernels is bounded: the grid barrier gives up after ~2^26
// polls, raises an error flag and the host reports NSG_ERR_TIMEOUT.
#include "nsg_internal.h"
#include "tagged.h"
#include "tuning_table.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>

namespace nsg {


static void raise_smem_limit(const void* fn, int bytes) { ensure_smem_limit(fn, bytes); }

namespace {

constexpr int kTriUnits = 1024;  // pass work units per CTA and step (columns x row blocks)

__device__ __forceinline__ double cre(double v) { return v; }
__device__ __forceinline__ double cre(double2 v) { return v.x; }
__device__ __forceinline__ double cabs2(double v) { return v * v; }
__device__ __forceinline__ double cabs2(double2 v) { return v.x * v.x + v.y * v.y; }
__device__ __forceinline__ double cconj(double v) { return v; }
__device__ __forceinline__ double2 cconj(double2 v) { return make_double2(v.x, -v.y); }
__device__ __forceinline__ double cmulv(double a, double b) { return a * b; }
__device__ __forceinline__ double2 cmulv(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double cscale(double a, double s) { return a * s; }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double cadd(double a, double b) { return a + b; }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double csub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
template <typename T>
__device__ __forceinline__ T czero();
template <>
__device__ __forceinline__ double czero<double>() { return 0.0; }
template <>
__device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }
template <typename T>
__device__ __forceinline__ T cone();
template <>
__device__ __forceinline__ double cone<double>() { return 1.0; }
template <>
__device__ __forceinline__ double2 cone<double2>() { return make_double2(1.0, 0.0); }

// v - a b - c d and acc + conj(a) b as chains of fused multiply-adds (two FP64
// operations per real element: the FP64 pipe bounds the tridiagonalisation)
__device__ __forceinline__ double fnms2(double v, double a, double b, double c, double d) {
  return fma(-c, d, fma(-a, b, v));
}
__device__ __forceinline__ double2 fnms2(double2 v, double2 a, double2 b, double2 c, double2 d) {
  double re = fma(c.y, d.y, fma(-c.x, d.x, fma(a.y, b.y, fma(-a.x, b.x, v.x))));
  double im = fma(-c.y, d.x, fma(-c.x, d.y, fma(-a.y, b.x, fma(-a.x, b.y, v.y))));
  return make_double2(re, im);
}
__device__ __forceinline__ double fcma(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ double2 fcma(double2 acc, double2 a, double2 b) {
  return make_double2(fma(a.y, b.y, fma(a.x, b.x, acc.x)), fma(-a.y, b.x, fma(a.x, b.y, acc.y)));
}

// acc + a b
__device__ __forceinline__ double cfma(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ double2 cfma(double2 acc, double2 a, double2 b) {
  return make_double2(fma(-a.y, b.y, fma(a.x, b.x, acc.x)), fma(a.y, b.x, fma(a.x, b.y, acc.y)));
}

// Grid barrier state of the tridiagonalisation (cooperative launch guarantees
// co-residency): a monotonic arrival counter (every CTA knows how many arrivals close
// each step, so nothing is reset between steps) and an error flag set by a wait that
// gave up.
struct Barrier {
  unsigned int count;
  int err;
};

// Householder scalars of a pivot column whose first entry below the diagonal is alpha
// and whose further entries have squared norm xnorm2: beta = -sign(Re alpha) times the
// column's norm, tau = (beta - alpha) / beta and the scale 1 / (alpha - beta) that turns
// the column into the reflector v (v[0] = 1).  A zero tail under a real alpha needs no
// reflection (tau = 0, beta = alpha).  By one warp, the quotients spread over lanes (each
// lane runs the same division on its own operands: one division sequence instead of two,
// or four for complex data); lane 0 stores the results.
template <typename T>
__device__ __forceinline__ void hh_scalars_warp(T alpha, double xnorm2, int lane, T& tk, T& scale, double& beta,
                                                bool& active) {
  // lane 0's operands for every lane: the branch below holds full-warp shuffles, so it
  // must be uniform over the warp whatever the caller's lanes hold
  xnorm2 = __shfl_sync(0xffffffffu, xnorm2, 0);
  const double ar = __shfl_sync(0xffffffffu, cre(alpha), 0);
  double ai = 0.0;
  if constexpr (sizeof(T) == 16) ai = __shfl_sync(0xffffffffu, ((double2&)alpha).y, 0);
  const bool act = !(xnorm2 == 0.0 && ai == 0.0);
  double bt = ar;
  T t = czero<T>(), s = czero<T>();
  if (act) {
    const double nrm = sqrt(ar * ar + ai * ai + xnorm2);
    bt = ar >= 0 ? -nrm : nrm;
    if constexpr (sizeof(T) == 16) {
      // tau = ((beta - ar) / beta, -ai / beta), scale = 1 / (ar - beta + i ai)
      const double zx = ar - bt, zy = ai;
      const double den = zx * zx + zy * zy;
      const double num = lane == 0 ? bt - ar : lane == 1 ? -ai : lane == 2 ? zx : -zy;
      const double dv = lane < 2 ? bt : den;
      const double qv = num / dv;
      const double q0 = __shfl_sync(0xffffffffu, qv, 0), q1 = __shfl_sync(0xffffffffu, qv, 1);
      const double q2 = __shfl_sync(0xffffffffu, qv, 2), q3 = __shfl_sync(0xffffffffu, qv, 3);
      double2 t2 = make_double2(q0, q1), s2 = make_double2(q2, q3);
      t = *(T*)&t2;
      s = *(T*)&s2;
    } else {
      const double qv = (lane == 0 ? bt - ar : 1.0) / (lane == 0 ? bt : ar - bt);
      const double q0 = __shfl_sync(0xffffffffu, qv, 0), q1 = __shfl_sync(0xffffffffu, qv, 1);
      t = *(T*)&q0;
      s = *(T*)&q1;
    }
  }
  if (lane == 0) {
    tk = t;
    scale = s;
    beta = bt;
    active = act;
  }
}

// The last subdiagonal entry has no reflector to make it real: for complex data its
// modulus is T's entry and its phase goes to *phase (the back-transformation multiplies
// the last row by it).
__device__ __forceinline__ double last_offdiagonal(double a, double2*) { return a; }
__device__ __forceinline__ double last_offdiagonal(double2 a, double2* phase) {
  const double r = hypot(a.x, a.y);
  *phase = r > 0 ? make_double2(a.x / r, a.y / r) : make_double2(1.0, 0.0);
  return r;
}

// Householder tridiagonalisation of the Hermitian n x n matrix A (column-major, both
// triangles stored).  On exit d[k] = T_kk, e[k] = T_k,k+1 (real), tau[k], the reflector
// vectors v_k (v_k[k+1] = 1 implicit) below the subdiagonal of column k.
// Step k: reflector from column k; x = tau A22 v; w = x - tau/2 (x^H v) v;
// A22 -= v w^H + w v^H.  The rank-2 update of step k-1 is applied lazily: every CTA
// rebuilds the updated pivot column itself, and one pass over the trailing block both
// applies the pending update and forms step k's x (one grid barrier per column).  CTAs
// retire as the trailing block shrinks (the barrier target follows the active count).
// A step is a chain of dependent L2 round trips, so the loads it needs are issued
// together: right after a barrier the next pivot column, x and the CTAs' partial sums,
// and at the top of a step the first tile of its pass.
template <typename T, int NT>
__global__ void __launch_bounds__(NT)
    tridiag_kernel(T* __restrict__ A, int n, double* __restrict__ d, double* __restrict__ e, T* __restrict__ tau,
                   T* __restrict__ xbuf, T* __restrict__ partial, Barrier* bar, int per_thread,
                   double2* __restrict__ phase) {
  extern __shared__ unsigned char smem_raw[];
  T* vprev = (T*)smem_raw;  // pending update (relative to rows >= k)
  T* wprev = vprev + n;
  T* vcur = wprev + n;      // current reflector (relative to rows >= k+1)
  __shared__ T red[NT / 32];
  __shared__ double2 wsum[NT / 32];
  __shared__ T part_s[kTriUnits];  // per-unit partial dot products of the pass
  __shared__ int s_ok;
  __shared__ T a0_s[kTriUnits];    // first entry (row k+1) of each own column after the update
  __shared__ T s_tk, s_scale, s_alpha2;  // the step's scalars, formed by one warp
  __shared__ double s_beta;
  __shared__ bool s_active;
  constexpr int nt = NT, nwarps = NT / 32;
  static_assert(nwarps >= 2 && (nwarps & (nwarps - 1)) == 0, "warp 0 plus pass warps, a power of two");
  constexpr bool cplx = sizeof(T) == 16;   // real data: the imaginary halves are never formed
  constexpr int P = (cplx ? 1024 : 2048) / NT;  // pivot-column and x entries per thread held in registers
  constexpr int PQ = 8;                      // CTA partial sums per lane held in registers
  constexpr int U = sizeof(T) == 8 ? 16 : 8, RB = 32 * U;
  const int tid = threadIdx.x, b = blockIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  bool has_prev = false;
  unsigned int target = 0;  // arrivals on the barrier counter that close the current step
  // step 0's pivot column as stored: rows 1 + tid + j nt, and the diagonal
  T raw[P];
  T rawd = czero<T>();
#pragma unroll
  for (int j = 0; j < P; ++j) {
    const int r = tid + j * nt;
    raw[j] = r < n - 1 ? __ldcg(A + 1 + r) : czero<T>();
  }
  if (b == 0 && tid == 0) rawd = __ldcg(A);
  for (int k = 0; k < n - 2; ++k) {
    const int m = n - k - 1;  // trailing size (rows k+1..n-1)
    // (32-bit index arithmetic: the order is at most ~8.5k, so m^2 and m x CTAs fit)
    int nact = (m * m + nt * per_thread - 1) / (nt * per_thread);
    nact = max(1, min(nact, (int)gridDim.x));
    if (b >= nact) return;
    // x and the partial sums are double-buffered by step parity: a CTA that runs ahead
    // writes the other buffer while a slower one still reads this step's values (the
    // barrier keeps every CTA within one step of the others)
    T* xb = xbuf + (size_t)(k & 1) * n;
    double2* pb = (double2*)partial + (size_t)(k & 1) * gridDim.x;
    // the CTA's columns [j0, j1) of the trailing block, in work units of one column x RB
    // rows dealt round-robin to the pass warps (every warp but warp 0, which forms the
    // step's scalars meanwhile: their chain of dependent FP64 operations would otherwise
    // delay warp 0's units); the block is final since the last barrier, so each pass
    // warp's first unit is requested before the pivot column is reduced
    const int j0 = m * b / nact, j1 = m * (b + 1) / nact;
    const int ncol = j1 - j0, nrb = (m + RB - 1) / RB, nunits = ncol * nrb;
    constexpr int PW = nwarps - 1;
    const int pw = warp - 1;
    T cur[U], nxt[U];
    auto load_unit = [&](int u, T* dst) {
      const int q = u / nrb, rb = u - q * nrb;
      const T* cj = A + (size_t)(k + 1 + j0 + q) * n + (k + 1);
#pragma unroll
      for (int t = 0; t < U; ++t) {
        const int r = rb * RB + 32 * t + lane;
        dst[t] = r < m ? __ldcg(cj + r) : czero<T>();
      }
    };
    if (warp > 0 && pw < nunits) load_unit(pw, cur);
    // 1. pivot column k with the pending update applied (rows k..n-1), reflector
    const T* colk = A + (size_t)k * n;
    const T wp0 = has_prev ? cconj(wprev[0]) : czero<T>();
    const T vp0 = has_prev ? cconj(vprev[0]) : czero<T>();
    T dk = czero<T>();
    if (b == 0 && tid == 0) dk = has_prev ? fnms2(rawd, vprev[0], wp0, wprev[0], vp0) : rawd;
    double ss = 0.0, ss1 = 0.0;  // two chains of dependent FP64 additions
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const int r = tid + j * nt;
      if (r < m) {
        T a = raw[j];
        if (has_prev) a = fnms2(a, vprev[r + 1], wp0, wprev[r + 1], vp0);
        vcur[r] = a;
        if (r > 0) {
          if (j & 1)
            ss1 += cabs2(a);
          else
            ss += cabs2(a);
        }
      }
    }
    ss += ss1;
    for (int r = tid + P * nt; r < m; r += nt) {  // orders above P nt + 1: loaded here
      T a = __ldcg(colk + k + 1 + r);
      if (has_prev) a = fnms2(a, vprev[r + 1], wp0, wprev[r + 1], vp0);
      vcur[r] = a;
      ss += cabs2(a);
    }
    // the squared norm: warp sums, then warp 0 adds them in warp order and forms the
    // reflector's scalars while the other warps start the pass (a warp-wide FP64
    // instruction holds a sub-partition's FP64 pipe for ~64 cycles on this GPU: the
    // scalar chain of square root and divides runs once per CTA, beside the pass).  The
    // pass needs no scalar: with v_0 = 1 and v_i = scale a_i (i > 0), where
    // alpha - beta = 1 / scale, A^H v = scale (A^H a - beta conj(A_0,:)); it forms A^H a
    // with the column as it is and keeps each column's first entry (a0_s).
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
    if (lane == 0) ((double*)red)[warp] = ss;
    __syncthreads();  // publishes vcur (the column a, unscaled) and the warp sums
    if (warp == 0) {
      // a tree over the warps' sums (lane 0 ends with the total; hh_scalars_warp takes
      // lane 0's operands for every lane)
      double xnorm2 = lane < nwarps ? ((double*)red)[lane] : 0.0;
      for (int o = nwarps / 2; o > 0; o >>= 1) xnorm2 += __shfl_xor_sync(0xffffffffu, xnorm2, o);
      hh_scalars_warp(vcur[0], xnorm2, lane, s_tk, s_scale, s_beta, s_active);
      if (b == 0 && lane == 0) {
        d[k] = cre(dk);
        e[k] = s_active ? s_beta : cre(vcur[0]);
        tau[k] = s_tk;
      }
    }
    // 2. the pass: pending update, then the dot products of the columns with a.  A warp
    //    loads its next unit before it updates and stores the current one (units are
    //    disjoint).  The trailing block is rewritten by other CTAs between steps: every
    //    access bypasses L1.
    T tk, scale;
    bool active;
    {
      for (int u = warp > 0 ? pw : nunits; u < nunits; u += PW) {
        if (u + PW < nunits) load_unit(u + PW, nxt);
        const int q = u / nrb, rb = u - q * nrb, jj = j0 + q;
        T* cj = A + (size_t)(k + 1 + jj) * n + (k + 1);
        const T wj = has_prev ? cconj(wprev[jj + 1]) : czero<T>();
        const T vj = has_prev ? cconj(vprev[jj + 1]) : czero<T>();
        T acc = czero<T>(), acc1 = czero<T>();
#pragma unroll
        for (int t = 0; t < U; ++t) {
          const int r = rb * RB + 32 * t + lane;
          if (r < m) {
            T val = cur[t];
            if (has_prev) {
              val = fnms2(val, vprev[r + 1], wj, wprev[r + 1], vj);
              __stcg(cj + r, val);
            }
            if (t == 0 && r == 0) a0_s[q] = val;
            if (t & 1)
              acc1 = fcma(acc1, val, vcur[r]);
            else
              acc = fcma(acc, val, vcur[r]);
          }
        }
        acc = cadd(acc, acc1);
        for (int o = 16; o > 0; o >>= 1) {
          if constexpr (sizeof(T) == 8) {
            acc += __shfl_down_sync(0xffffffffu, acc, o);
          } else {
            double2 t2;
            t2.x = __shfl_down_sync(0xffffffffu, ((double2&)acc).x, o);
            t2.y = __shfl_down_sync(0xffffffffu, ((double2&)acc).y, o);
            acc = cadd(acc, *(T*)&t2);
          }
        }
        if (lane == 0) part_s[u] = acc;
#pragma unroll
        for (int t = 0; t < U; ++t) cur[t] = nxt[t];
      }
      __syncthreads();  // publishes the partial sums, a0_s and the scalars
      tk = s_tk;
      scale = s_scale;
      active = s_active;
      const double beta = s_beta;
      const T ts = cmulv(tk, scale);
      // column sums in a fixed order, x, and this CTA's share of x^H v (a warp whose
      // threads own no column contributes nothing and skips its reduction)
      const int cwarps = (ncol + 31) / 32;
      if (warp < cwarps) {
        double2 pacc = make_double2(0.0, 0.0);
        for (int q = tid; q < ncol; q += nt) {
          T sum = czero<T>();
          for (int rb = 0; rb < nrb; ++rb) sum = cadd(sum, part_s[q * nrb + rb]);
          const T xi = cmulv(ts, csub(sum, cscale(cconj(a0_s[q]), beta)));
          __stcg(xb + j0 + q, xi);
          const T vq = (j0 + q == 0) ? cone<T>() : cmulv(scale, vcur[j0 + q]);
          const T p = cmulv(cconj(xi), vq);
          if constexpr (!cplx) {
            pacc.x += (double&)p;
          } else {
            pacc.x += ((double2&)p).x;
            pacc.y += ((double2&)p).y;
          }
        }
        for (int o = 16; o > 0; o >>= 1) {
          pacc.x += __shfl_down_sync(0xffffffffu, pacc.x, o);
          if constexpr (cplx) pacc.y += __shfl_down_sync(0xffffffffu, pacc.y, o);
        }
        if (lane == 0) wsum[warp] = pacc;
      }
      __syncthreads();
      // the reflector v itself (v_0 = 1) for the update, its storage and the next step
      for (int r = tid; r < m; r += nt) vcur[r] = (r == 0) ? cone<T>() : cmulv(vcur[r], scale);
      if (tid == 0) {
        double2 sacc = cwarps > 0 ? wsum[0] : make_double2(0.0, 0.0);
        for (int w = 1; w < cwarps; ++w) {
          sacc.x += wsum[w].x;
          if constexpr (cplx) sacc.y += wsum[w].y;
        }
        __stcg(pb + b, sacc);
      }
    }
    // 3. barrier among the active CTAs: every CTA active now was active in every earlier
    //    step (the active count never grows), so all of them agree on the target
    target += unsigned(nact);
    __syncthreads();
    if (tid == 0) {
      // arrival with release semantics (the block barrier above orders every thread's
      // stores of this step before it), polling with acquire semantics (the peers' stores
      // are visible after it, and the block barrier below passes that on): the same
      // ordering as full fences on both sides, without their cost
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&bar->count), "r"(1u) : "memory");
      long long polls = 0;
      for (;;) {
        unsigned int cnt;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cnt) : "l"(&bar->count) : "memory");
        if (int(cnt - target) >= 0) break;
        if (++polls > (1ll << 26) || *(volatile int*)&bar->err) {
          atomicExch(&bar->err, 1);
          break;
        }
        __nanosleep(20);
      }
      s_ok = (*(volatile int*)&bar->err) == 0;
    }
    __syncthreads();
    if (!s_ok) return;
    // 4. requested together: x, the CTAs' partials of x^H v, and the next pivot column
    //    (column k+1: rows k+2.. and its diagonal) as the pass above stored it
    T xr[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const int r = tid + j * nt;
      xr[j] = r < m ? __ldcg(xb + r) : czero<T>();
    }
    double2 pq[PQ];
    if (warp == 0) {
#pragma unroll
      for (int j = 0; j < PQ; ++j) {
        const int q = lane + 32 * j;
        pq[j] = q < nact ? __ldcg(pb + q) : make_double2(0.0, 0.0);
      }
    }
    {
      const T* coln = A + (size_t)(k + 1) * n + (k + 2);
#pragma unroll
      for (int j = 0; j < P; ++j) {
        const int r = tid + j * nt;
        raw[j] = r < m - 1 ? __ldcg(coln + r) : czero<T>();
      }
      if (b == 0 && tid == 0) rawd = __ldcg(A + (size_t)(k + 1) * n + (k + 1));
    }
    for (int r = tid + P * nt; r < m; r += nt) wprev[r] = __ldcg(xb + r);
    // warp 0 sums the CTAs' partials (lane-strided in ascending order, then a butterfly:
    // the same value in every CTA) and forms alpha2 for the CTA
    if (warp == 0) {
      // a tree over the lane's partials, then over the lanes
#pragma unroll
      for (int h = PQ / 2; h > 0; h >>= 1)
#pragma unroll
        for (int j = 0; j < h; ++j) {
          pq[j].x += pq[j + h].x;
          if constexpr (cplx) pq[j].y += pq[j + h].y;
        }
      double2 xv = pq[0];
      for (int q = lane + 32 * PQ; q < nact; q += 32) {
        const double2 t = __ldcg(pb + q);
        xv.x += t.x;
        if constexpr (cplx) xv.y += t.y;
      }
      for (int o = 16; o > 0; o >>= 1) {
        xv.x += __shfl_xor_sync(0xffffffffu, xv.x, o);
        if constexpr (cplx) xv.y += __shfl_xor_sync(0xffffffffu, xv.y, o);
      }
      if (lane == 0) {
        T xvT;
        if constexpr (sizeof(T) == 8) {
          double t1 = xv.x;
          xvT = *(T*)&t1;
        } else {
          xvT = *(T*)&xv;
        }
        s_alpha2 = cscale(cmulv(tk, xvT), -0.5);
      }
    }
    __syncthreads();
    const T alpha2 = s_alpha2;
    // reflector storage below the subdiagonal of column k: every CTA has read column k
    // before the barrier, and it is not read again
    if (b == 0)
      for (int r = tid + 1; r < m; r += nt) A[(size_t)k * n + (k + 1 + r)] = vcur[r];
    // 5. w = x + alpha2 v becomes the pending update (relative to rows >= k+1); a thread
    //    rewrites only the entries it holds
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const int r = tid + j * nt;
      if (r < m) {
        vprev[r] = vcur[r];
        wprev[r] = active ? cadd(xr[j], cmulv(alpha2, vcur[r])) : czero<T>();
      }
    }
    for (int r = tid + P * nt; r < m; r += nt) {
      vprev[r] = vcur[r];
      wprev[r] = active ? cadd(wprev[r], cmulv(alpha2, vcur[r])) : czero<T>();
    }
    has_prev = active;
    __syncthreads();
  }
  if (b == 0 && tid == 0) {
    // last 2 x 2 block with the pending update of step n-3 (relative to rows >= n-2)
    auto upd = [&](int i, int j) -> T {
      T a = __ldcg(A + i + (size_t)j * n);
      if (has_prev && n >= 3)
        a = csub(a, cadd(cmulv(vprev[i - (n - 2)], cconj(wprev[j - (n - 2)])),
                         cmulv(wprev[i - (n - 2)], cconj(vprev[j - (n - 2)]))));
      return a;
    };
    if (n >= 2) {
      T a11 = upd(n - 2, n - 2), a21 = upd(n - 1, n - 2), a22 = upd(n - 1, n - 1);
      d[n - 2] = cre(a11);
      e[n - 2] = last_offdiagonal(a21, phase);
      d[n - 1] = cre(a22);
    } else {
      d[0] = cre(A[0]);
    }
  }
}

// Householder tridiagonalisation with the matrix resident in shared memory: column j lives
// in CTA j mod C for the whole reduction, so a step moves only one row of the matrix and the
// vector x between SMs.  The CTAs are one thread-block cluster (both pushed to the peers'
// shared memory, one cluster barrier per step) or, GRID, up to one per SM (exchanged through
// L2 in 16-byte pieces that carry the step's number beside the value, so a consumer polls the
// data itself: no counter, no fence, and no second round trip for the data after a barrier).
// Same reflectors, tau, d and e as tridiag_kernel.
//
// Step k, with the rank-2 update of step k-1 pending (reflector v, x = tau A v):
//   p = Re x^H v,  c = -|tau|^2 / Re(tau) p,  w'_j = x_j + c v_j:  A -= v w'^H + x v^H
//   (the usual w = x + c/2 v enters both products; here all of c v v^H goes to the first, so
//   w' is needed only at the CTA's own columns);
//   a = the pivot column with the update applied, in every CTA (same data, same order);
//   one pass over the own trailing columns applies the update and forms S_j = A[:, j]^H a;
//   x_j = conj(A_k+1,j) - S_j / beta, sent with A_k+1,j, which the others take as the next
//   pivot column (A is Hermitian).
// v = scale a but for v_0 = 1, and tau scale = -1 / beta: the new x needs a reciprocal square
// root and nothing else, and the column a is kept as it is, with scale in the coefficients.
// A thread keeps the same rows (from the last one up, so that finished rows leave whole
// iterations) through every phase of a step, so the vectors need no barrier of their own.
//
// Bound: the dependent chain of a step (gather, sum, pivot column, pass, publication; about
// 5500 cycles at order 128), and from about order 700 the FP64 pipe (3 operations an
// element).  An FP64 instruction of a warp holds its SM sub-partition for 64 cycles whatever
// its active lanes, so the count of such instructions on the chain is what costs: one pass
// warp per sub-partition (it fills the pipe with independent elements, and leaves less to sum
// over the CTA), a further warp for the sums and scalars beside the pass, no loop unrolled
// past the rows a thread has.  us per column, over all SMs against tridiag_kernel (above
// order 384) or a cluster that read the pivot column and x from its peers in two barriers a
// step: real order 128 2.8 / 4.2, 256 3.2 / 5.7, 512 4.4 / 7.8, 950 6.9 / 9.3; complex 128
// 4.3 / 6.9, 256 6.1 / 11.9, 950 15.9 / 25.3.  One cluster: real 24 3.3 / 3.9, 64 3.2 / 3.8.
// (Tried and slower: sums in exact integer arithmetic, 1050 cycles against 720 by shuffles;
// the messages in several copies; x and the pivot column interleaved, twice the sectors.)
constexpr int kResWarps = 4;                // pass warps
constexpr int kResPass = 32 * kResWarps;    // pass threads
constexpr int kResThreads = kResPass + 32;  // and the scalar warp
constexpr int kResCols = 128;               // own columns of a CTA, at most
constexpr int kPollDelay = 500;             // cycles between publishing and the first poll (order
                                            // 256: 820 us, with none 1380, 300 875, 800 845)

// row r's message, S_r and the next pivot column's entry, in two runs of n rows
__device__ __forceinline__ void put_row(ulonglong2* buf, int n, int r, double S, double a, unsigned long long tag) {
  put_tagged(buf + r, S, tag);
  put_tagged(buf + n + r, a, tag);
}
__device__ __forceinline__ void put_row(ulonglong2* buf, int n, int r, double2 S, double2 a, unsigned long long tag) {
  put_tagged(buf + 2 * r, S.x, tag);
  put_tagged(buf + 2 * r + 1, S.y, tag);
  put_tagged(buf + 2 * (n + r), a.x, tag);
  put_tagged(buf + 2 * (n + r) + 1, a.y, tag);
}
__device__ __forceinline__ bool get_row(const ulonglong2* buf, int n, int r, unsigned long long tag, double& S, double& a) {
  const bool k0 = get_tagged(buf + r, tag, S), k1 = get_tagged(buf + n + r, tag, a);
  return k0 && k1;
}
__device__ __forceinline__ bool get_row(const ulonglong2* buf, int n, int r, unsigned long long tag, double2& S, double2& a) {
  const bool k0 = get_tagged(buf + 2 * r, tag, S.x), k1 = get_tagged(buf + 2 * r + 1, tag, S.y);
  const bool k2 = get_tagged(buf + 2 * (n + r), tag, a.x), k3 = get_tagged(buf + 2 * (n + r) + 1, tag, a.y);
  return k0 && k1 && k2 && k3;
}
__device__ __forceinline__ double shfl_x(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double2 shfl_x(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
// x + c v for a real c
__device__ __forceinline__ double caxpy(double c, double v, double x) { return fma(c, v, x); }
__device__ __forceinline__ double2 caxpy(double c, double2 v, double2 x) {
  return make_double2(fma(c, v.x, x.x), fma(c, v.y, x.y));
}
// v - a b
__device__ __forceinline__ double cfnma(double v, double a, double b) { return fma(-a, b, v); }
__device__ __forceinline__ double2 cfnma(double2 v, double2 a, double2 b) {
  return make_double2(fma(a.y, b.y, fma(-a.x, b.x, v.x)), fma(-a.y, b.x, fma(-a.x, b.y, v.y)));
}
// s + |a|^2
__device__ __forceinline__ double sqacc(double s, double a) { return fma(a, a, s); }
__device__ __forceinline__ double sqacc(double s, double2 a) { return fma(a.y, a.y, fma(a.x, a.x, s)); }

// barriers between the pass warps and the scalar warp: a side that has nothing to wait for
// only arrives
__device__ __forceinline__ void bar_sync(int id, int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ bool not_zero(double a) { return (__double_as_longlong(a) << 1) != 0; }
__device__ __forceinline__ bool not_zero(double2 a) { return not_zero(a.x) || not_zero(a.y); }

// The pass over NB own columns from cols: update, dot products with a, and their sums over
// the warp (part[b]; the values are reduced together: the first levels of the butterfly halve
// those a lane holds, so that eight take 9 additions).  Rows rtop, rtop - kResPass, .. rlow.
template <typename T, int NB>
__device__ __forceinline__ void resident_pass(T* cols, int n, const T* wpc, const T* vpc, const T* uu, const T* xx,
                                              const T* aa, int rtop, int rlow, int lane, T* part) {
  constexpr int NP = NB > 4 ? 8 : NB > 2 ? 4 : NB;  // rounded to a power of two
  T w[NB], v0[NB], acc[NP], nxt[NB];
#pragma unroll
  for (int b = 0; b < NP; ++b) acc[b] = czero<T>();
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    w[b] = wpc[b];
    v0[b] = vpc[b];
    nxt[b] = rtop >= rlow ? cols[(size_t)b * n + rtop] : czero<T>();
  }
  for (int r = rtop; r >= rlow; r -= kResPass) {
    T val[NB];
    const T ur = uu[r], xr = xx[r], ar = aa[r];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      val[b] = nxt[b];
      if (r - kResPass >= rlow) nxt[b] = cols[(size_t)b * n + r - kResPass];
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) val[b] = fnms2(val[b], ur, w[b], xr, v0[b]);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      acc[b] = fcma(acc[b], val[b], ar);
      cols[(size_t)b * n + r] = val[b];
    }
  }
  int o = 16;
#pragma unroll
  for (int h = NP / 2; h >= 1; h /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const T send = up ? acc[i] : acc[i + h], keep = up ? acc[i + h] : acc[i];
      acc[i] = cadd(keep, shfl_x(send, o));
    }
  }
  for (; o > 0; o /= 2) acc[0] = cadd(acc[0], shfl_x(acc[0], o));
  constexpr int kLow = 32 / NP;  // lanes that hold the same column's sum
  if (lane % kLow == 0 && lane / kLow < NB) part[lane / kLow] = acc[0];
}

// A thread's rows of the messages with tag k, PU requested together; scalars() once, before
// the first row is taken.  False when the wait gives up.
template <typename T, int PU, typename Scalars, typename Take>
__device__ __forceinline__ bool resident_gather(const ulonglong2* in, int n, int rtop, int k, Barrier* bar,
                                                Scalars scalars, Take take) {
  bool good = true, first = true;
  for (int r0 = rtop; first || r0 >= k; r0 -= PU * kResPass, first = false) {
    T S[PU], raw[PU];
    for (int polls = 0;; ++polls) {
      bool ok = true;
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        const int r = r0 - u * kResPass;
        if (r >= k) ok = get_row(in, n, r, (unsigned long long)k, S[u], raw[u]) && ok;
      }
      if (ok) break;
      if (polls > (1 << 22) || ((polls & 255) == 255 && *(volatile int*)&bar->err)) {
        atomicExch(&bar->err, 1);
        good = false;
        break;
      }
    }
    if (first) scalars();
#pragma unroll
    for (int u = 0; u < PU; ++u) {
      const int r = r0 - u * kResPass;
      if (r >= k) take(r, S[u], raw[u]);
    }
  }
  return good;
}

template <typename T, bool GRID>
__global__ void __launch_bounds__(kResThreads)
    tridiag_resident_kernel(T* __restrict__ A, int n, double* __restrict__ d, double* __restrict__ e,
                            T* __restrict__ tau, double2* __restrict__ phase, ulonglong2* xch, Barrier* bar) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int C = GRID ? int(gridDim.x) : int(cluster.num_blocks());
  const int rank = GRID ? int(blockIdx.x) : int(cluster.block_rank());
  const int ncol = (n - rank + C - 1) / C;  // columns j = rank + C q, q < ncol
  const int ncmax = (n + C - 1) / C;        // the layout is the same in every CTA (peers address it)
  constexpr bool cplx = sizeof(T) == 16;
  constexpr int kBatch = cplx ? 4 : 8;      // columns of one pass over the rows
  constexpr int kScalars = 1, kSum = 2, kUpdate = 3, kNorm = 4, kColumns = 5;  // barriers
  extern __shared__ __align__(16) unsigned char ct_smem[];
  T* cols = (T*)ct_smem;               // own columns, n rows each
  T* abuf = cols + (size_t)ncmax * n;  // pivot columns of this step and the last, by step parity
  T* xg = abuf + 2 * n;                // x; with the peers as writers of S by step parity, then
                                       // the next pivot column likewise
  __shared__ double psum[2][kResPass];
  __shared__ T part[kResWarps][kResCols], wpc[kResCols], vpc[kResCols];
  __shared__ T s_w0, s_scale;
  __shared__ double s_c, s_f;
  __shared__ int s_fail, s_tail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool scalar_warp = warp == kResWarps;
  // the thread's rows: rtop - i kResPass; the last rows to the last pass warp, so that the
  // warp beside the scalar warp on its sub-partition has the fewest
  const int rtop = n - 1 - (tid ^ (kResPass - 32));
  for (int q = 0; q < ncol; ++q) {
    const T* src = A + (size_t)(rank + C * q) * n;
    for (int r = tid; r < n; r += kResThreads) cols[(size_t)q * n + r] = src[r];
  }
  for (int r = tid; r < n; r += kResThreads) abuf[n + r] = czero<T>();  // no update is pending at step 0
  if (tid == 0) s_fail = s_tail = 0;
  // the scalar warp's state of the pending update: scale, ctau = |tau|^2 / Re(tau) and
  // m1 = -ctau scale
  T scale = czero<T>(), m1 = czero<T>();
  double ctau = 0.0;
  if constexpr (GRID)
    __syncthreads();
  else
    cluster.sync();
  auto warp_sum = [&](const double* v) {  // of kResPass values, on every lane of the scalar warp
    static_assert(kResPass == 128, "four values per lane");
    double s = (v[lane] + v[lane + 32]) + (v[lane + 64] + v[lane + 96]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  };
  for (int k = 0; k < n - 1; ++k) {
    const int q0 = (k + 1 - rank + C - 1) / C, nown = ncol - q0;  // own trailing columns (j > k)
    const bool last = k == n - 2;  // the final 2 x 2 block: nothing left to reflect
    if (nown <= 0) {
      if constexpr (GRID) return;
      if (!last) cluster.sync();
      continue;
    }
    const bool stores = rank == min(k + 1 + C / 2, n - 1) % C;  // this step's results are written by one CTA
    T* aa = abuf + (k & 1) * n;
    T* uu = abuf + ((k + 1) & 1) * n;
    T* xx = GRID ? xg : xg + ((k + 1) & 1) * n;
    if (scalar_warp) {
      // c = -ctau (Re x_k + Re scale sum conj(x) a), and scale conj(w') at the own columns and
      // (the last lane) at the pivot, whose v is 1; what does not need x comes before the wait
      const bool at_pivot = lane == 31;
      T vj = czero<T>(), sv = czero<T>();
      int j = k;
      auto own = [&](int q) {
        j = rank + C * (q0 + q);
        vj = cconj(cmulv(scale, uu[j]));
        sv = cmulv(scale, vj);
      };
      if (at_pivot)
        sv = scale;
      else if (lane < nown)
        own(lane);
      bar_sync(kSum, kResThreads);
      if (GRID && s_fail) {
        bar_arrive(kUpdate, kResThreads);
        return;
      }
      const double m0 = -ctau * cre(xx[k]);
      T xj = cmulv(scale, cconj(xx[j]));
      double c;
      if constexpr (cplx)
        c = fma(m1.x, warp_sum(psum[0]), fma(-m1.y, warp_sum(psum[1]), m0));
      else
        c = fma(m1, warp_sum(psum[0]), m0);
      {
        const T w = caxpy(c, sv, xj);
        if (at_pivot) {
          s_w0 = w;
          s_c = c;
        } else if (lane < nown) {
          vpc[lane] = vj;
          wpc[lane] = w;
        }
      }
      for (int q = 31 + lane; q < nown; q += 32) {
        own(q);
        vpc[q] = vj;
        wpc[q] = caxpy(c, sv, cmulv(scale, cconj(xx[j])));
      }
      bar_arrive(kUpdate, kResThreads);
      // the scalars of column k's reflector, beside the pass
      bar_sync(kNorm, kResThreads);
      const T alpha = aa[k + 1];
      if (last) {
        if (stores && lane == 0) e[k] = last_offdiagonal(alpha, phase);
        break;
      }
      const double x2 = warp_sum(psum[0]), ar = cre(alpha);
      double ai = 0.0;
      if constexpr (cplx) ai = alpha.y;
      // (a norm whose square is subnormal has lost its digits, and H its orthogonality)
      const bool active = __double2hiint(x2) >= 0x00100000 && (s_tail || not_zero(ai));
      const double rr = active ? rsqrt(x2) : 0.0;
      const bool neg = __double2hiint(ar) < 0;
      __syncwarp();
      if (lane == 0) {
        s_f = neg ? -rr : rr;  // -1 / beta, or 0 for no reflection
        s_tail = 0;
      }
      bar_arrive(kScalars, kResThreads);
      T tk = czero<T>();
      double beta = ar;
      scale = czero<T>();
      ctau = 0.0;
      if (active) {
        double nrm = x2 * rr;
        nrm = fma(0.5 * rr, fma(-nrm, nrm, x2), nrm);
        const double sg = neg ? -1.0 : 1.0, big = fabs(ar) + nrm;  // alpha - beta = (sg big, ai)
        beta = neg ? nrm : -nrm;
        if constexpr (cplx) {
          const double inv = 1.0 / fma(ai, ai, big * big);
          scale = make_double2(sg * big * inv, -ai * inv);
          tk = make_double2(fma(fabs(ar), rr, 1.0), sg * ai * rr);
          ctau = (tk.x * tk.x + tk.y * tk.y) / tk.x;
        } else {
          scale = sg / big;
          tk = fma(fabs(ar), rr, 1.0);
          ctau = tk;
        }
      }
      m1 = cscale(scale, -ctau);
      if (lane == 0) {
        s_scale = scale;
        if (stores) {
          e[k] = beta;
          tau[k] = tk;
        }
      }
      if constexpr (!GRID) cluster.sync();
      continue;
    }
    // 1. the pending update's x; sum of conj(x) a
    T p = czero<T>();
    double f = 0.0;
    auto take = [&](int r, T S, T raw) {
      const T x = not_zero(f) ? caxpy(f, S, raw) : czero<T>();
      xx[r] = x;
      aa[r] = not_zero(f) ? S : raw;
      if (r > k) p = fcma(p, x, uu[r]);
    };
    if (k == 0) {
      for (int r = rtop; r >= 0; r -= kResPass) take(r, czero<T>(), A[r]);
    } else if constexpr (GRID) {
      const ulonglong2* in = xch + (size_t)((k + 1) & 1) * (cplx ? 4 : 2) * n;
      // polls that come before the messages slow down the stores they wait for
      for (const long long t0 = clock64(); clock64() - t0 < kPollDelay;) {
      }
      bool ok = true;
      const int nr = (n - k + kResPass - 1) / kResPass;  // rows of a thread, at most
      auto scalars = [&] {
        bar_sync(kScalars, kResThreads);
        f = s_f;
      };
      if (nr == 1)
        ok = resident_gather<T, 1>(in, n, rtop, k, bar, scalars, take);
      else if (nr == 2)
        ok = resident_gather<T, 2>(in, n, rtop, k, bar, scalars, take);
      else if (nr <= 4 || cplx)
        ok = resident_gather<T, 4>(in, n, rtop, k, bar, scalars, take);
      else
        ok = resident_gather<T, cplx ? 4 : 8>(in, n, rtop, k, bar, scalars, take);
      if (!ok) s_fail = 1;
    } else {
      bar_sync(kScalars, kResThreads);
      f = s_f;
      const T* raw = xg + (2 + ((k + 1) & 1)) * n;
      for (int r = rtop; r >= k; r -= kResPass) take(r, xx[r], raw[r]);
    }
    if constexpr (cplx) {
      psum[0][tid] = p.x;
      psum[1][tid] = p.y;
    } else {
      psum[0][tid] = p;
    }
    bar_arrive(kSum, kResThreads);
    // 2. the pivot column: A_r,k - x_r = -f S_r without the term in v (v_k = 1), which comes
    //    with c; its squared norm
    if (not_zero(f))
      for (int r = rtop; r >= k; r -= kResPass) aa[r] = cscale(aa[r], -f);
    bar_sync(kUpdate, kResThreads);
    if (GRID && s_fail) return;
    const T w0 = s_w0, sc = s_scale;
    bool tail = false;
    double ss = 0.0;
    for (int r = rtop; r > k; r -= kResPass) {
      const T a = cfnma(aa[r], uu[r], w0);
      aa[r] = a;
      ss = sqacc(ss, a);
      tail = tail || (r > k + 1 && not_zero(a));
    }
    psum[0][tid] = ss;
    if (tail) s_tail = 1;
    bar_arrive(kNorm, kResThreads);
    // 3. the pass over the own columns
    const bool rows = n - 1 - 32 * (kResWarps - 1 - warp) > k;  // does the warp hold trailing rows?
    const int nbat = (nown + kBatch - 1) / kBatch, per = (nown + nbat - 1) / nbat;
    for (int q = 0; q < nown; q += per) {
      T* cq = cols + (size_t)(q0 + q) * n;
      const int nb = min(per, nown - q);
      if (!rows) {
        if (lane < nb) part[warp][q + lane] = czero<T>();
        continue;
      }
#define NSG_RESIDENT_PASS(NB) \
  case NB:                    \
    resident_pass<T, NB>(cq, n, wpc + q, vpc + q, uu, xx, aa, rtop, k + 1, lane, &part[warp][q]); \
    break
      switch (nb) {
        NSG_RESIDENT_PASS(1);
        NSG_RESIDENT_PASS(2);
        NSG_RESIDENT_PASS(3);
        NSG_RESIDENT_PASS(4);
        default:
          if constexpr (!cplx) {
            switch (nb) {
              NSG_RESIDENT_PASS(5);
              NSG_RESIDENT_PASS(6);
              NSG_RESIDENT_PASS(7);
              NSG_RESIDENT_PASS(8);
            }
          }
      }
#undef NSG_RESIDENT_PASS
    }
    if (last) {
      if (rtop == n - 1) d[n - 1] = cre(cols[(size_t)(ncol - 1) * n + n - 1]);
    } else {
      bar_sync(kColumns, kResPass);
      // 4. S and row k+1 at the own columns, to everyone
      auto sum_of = [&](int q, T& a0) {
        static_assert(kResWarps == 4, "the tree below");
        a0 = cconj(cols[(size_t)(q0 + q) * n + k + 1]);
        return cadd(cadd(part[0][q], part[1][q]), cadd(part[2][q], part[3][q]));
      };
      if constexpr (GRID) {
        ulonglong2* out = xch + (size_t)(k & 1) * (cplx ? 4 : 2) * n;
        for (int q = tid; q < nown; q += kResPass) {
          T a0;
          const T S = sum_of(q, a0);
          put_row(out, n, rank + C * (q0 + q), S, a0, (unsigned long long)(k + 1));
        }
      } else {
        for (int i = tid; i < nown * C; i += kResPass) {
          const int q = i / C, peer = i - q * C, j = rank + C * (q0 + q);
          T a0;
          const T S = sum_of(q, a0);
          T* out = cluster.map_shared_rank(xg, peer) + (k & 1) * n;
          out[j] = S;
          out[2 * n + j] = a0;
        }
        cluster.barrier_arrive();
      }
    }
    // d_k, and the last reflector to its place below the subdiagonal of column k-1 (column 0
    // of A has been read by every CTA: each has published since)
    if (stores) {
      if ((rtop - k) % kResPass == 0) d[k] = cre(aa[k]) - (cre(xx[k]) + s_c);  // the thread that holds row k
      if (k > 0) {
        T* gcol = A + (size_t)(k - 1) * n;
        for (int r = rtop; r > k; r -= kResPass) gcol[r] = cmulv(uu[r], sc);
      }
    }
    if (last) break;
    if constexpr (!GRID) cluster.barrier_wait();
  }
  if constexpr (!GRID) cluster.sync();  // no CTA leaves while another may still write its shared memory
}

// Eigenvectors first, first + step, ... of T (columns of Q) as the columns of Z, the last
// row times the phase of T's last subdiagonal entry.
__global__ void gather_vectors_kernel(const double* __restrict__ Q, int64_t n, int64_t first, int64_t step,
                                      int64_t count, double* __restrict__ Z, int64_t ldz, const double2*) {
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n * count; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e % n, j = e / n;
    Z[i + j * ldz] = Q[i + (first + j * step) * n];
  }
}
__global__ void gather_vectors_kernel(const double* __restrict__ Q, int64_t n, int64_t first, int64_t step,
                                      int64_t count, double2* __restrict__ Z, int64_t ldz, const double2* phase) {
  const double2 ph = *phase;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < n * count; e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = e % n, j = e / n;
    const double v = Q[i + (first + j * step) * n];
    Z[i + j * ldz] = i == n - 1 ? make_double2(ph.x * v, ph.y * v) : make_double2(v, 0.0);
  }
}

// compact WY: T factors of all reflector blocks in one launch (block b = CTA b; kWY = 64
// reflectors per block, zero-padded with tau = 0) from S_b = V_b^H V_b, by doubling: with the
// factors T1, T2 of two neighbouring halves, T = [T1, -T1 S12 T2; 0, T2].  Each level is two
// triangular products over all pairs at once, so the 64^3 / 6 multiply-adds spread over the
// CTA's FP64 pipes (column by column, one thread per row, they were a chain of 119 us for
// real and 483 us for complex data; this takes 34 and 94).
constexpr int kWY = 64, kWYThreads = 512;
template <typename T>
__global__ void __launch_bounds__(kWYThreads) wy_tfactor_kernel(const T* S, const T* tau, T* Tm) {
  extern __shared__ __align__(16) unsigned char wy_smem[];  // 2 x kWY x (kWY + 1) elements
  T(*Ss)[kWY + 1] = (T(*)[kWY + 1])wy_smem;  // [column][row]; the pairs' S12 T2 replaces S12
  T(*Ts)[kWY + 1] = Ss + kWY;                // [column][row]
  const int tid = threadIdx.x, b = blockIdx.x;
  const T* Sb = S + (size_t)b * kWY * kWY;
  T* Tb = Tm + (size_t)b * kWY * kWY;
  for (int t = tid; t < kWY * kWY; t += kWYThreads) {
    const int i = t % kWY, j = t / kWY;
    Ss[j][i] = Sb[t];
    Ts[j][i] = i == j ? tau[(size_t)b * kWY + i] : czero<T>();
  }
  __syncthreads();
  for (int h = 1; h < kWY; h *= 2) {
    // output (i, j) of pair q: row i of its upper half, column j of its lower half
    constexpr int NI = kWY * kWY / 4 / kWYThreads;  // outputs per thread, at the last level
    T acc[NI];
#pragma unroll
    for (int x = 0; x < NI; ++x) {
      const int t = tid + x * kWYThreads, i = t % h, j = t / h % h, q = t / (h * h);
      acc[x] = czero<T>();
      if (q < kWY / (2 * h)) {
        const int r0 = 2 * h * q, c0 = r0 + h;
        for (int l = 0; l <= j; ++l) acc[x] = cfma(acc[x], Ss[c0 + l][r0 + i], Ts[c0 + j][c0 + l]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < NI; ++x) {
      const int t = tid + x * kWYThreads, i = t % h, j = t / h % h, q = t / (h * h);
      if (q < kWY / (2 * h)) Ss[2 * h * q + h + j][2 * h * q + i] = acc[x];
    }
    __syncthreads();
    for (int t = tid; t < kWY / 2 * h; t += kWYThreads) {
      const int i = t % h, j = t / h % h, r0 = 2 * h * (t / (h * h)), c0 = r0 + h;
      T sum = czero<T>();
      for (int l = i; l < h; ++l) sum = cfma(sum, Ts[r0 + l][r0 + i], Ss[c0 + j][r0 + l]);
      Ts[c0 + j][r0 + i] = cscale(sum, -1.0);
    }
    __syncthreads();
  }
  for (int t = tid; t < kWY * kWY; t += kWYThreads) Tb[t] = Ts[t / kWY][t % kWY];
}

// all reflectors as the columns of an n x ncols matrix (v_kk[kk+1] = 1, zeros above,
// zero columns beyond the last reflector)
template <typename T>
__global__ void wy_extract_all_kernel(const T* A, int n, int nref, int ncols, T* V) {
  const size_t tot = (size_t)n * ncols;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int r = int(e % n), kk = int(e / n);
    T val = czero<T>();
    if (kk < nref) {
      if (r == kk + 1)
        val = cone<T>();
      else if (r > kk + 1)
        val = A[r + (size_t)kk * n];
    }
    V[e] = val;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------

struct DevBuf {
  nsg_ctx* c;
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf(nsg_ctx* cc, size_t b) : c(cc), bytes(b) { p = dalloc(c, b); }
  ~DevBuf() { dfree(c, p, bytes); }
  template <typename T>
  T* as() {
    return (T*)p;
  }
};

// Back-transformation Z <- H_0 H_1 ... H_{n-3} Z in blocks of kWY reflectors, last block
// first.  Every block's V, S = V^H V and T factor are formed up front (one launch each,
// before the eigenvalues are known on the host); the sequential part is then three GEMMs
// per block.
template <typename T>
struct BackTransform {
  nsg_ctx* c;
  const int dtype, n, nref, NB, nblk, ncols;
  DevBuf V, S, Tm, taup;
  BackTransform(nsg_ctx* cc, int dt, int order, const T* A, const T* tau_dev);
  void apply(T* Z, int64_t ldz, int64_t k);
};

template <typename T>
BackTransform<T>::BackTransform(nsg_ctx* cc, int dt, int order, const T* A, const T* tau_dev)
    : c(cc),
      dtype(dt),
      n(order),
      nref(std::max(order - 2, 0)),
      NB(kWY),
      nblk((nref + kWY - 1) / kWY),
      ncols(nblk * kWY),
      V(cc, sizeof(T) * (size_t)order * ncols),
      S(cc, sizeof(T) * (size_t)kWY * kWY * nblk),
      Tm(cc, sizeof(T) * (size_t)kWY * kWY * nblk),
      taup(cc, sizeof(T) * ncols) {
  if (nref == 0) return;
  const size_t eb = sizeof(T);
  {
    int gblocks = int(std::min<size_t>(((size_t)n * ncols + 255) / 256, (size_t)c->num_sms * 8));
    wy_extract_all_kernel<T><<<gblocks, 256, 0, c->stream>>>(A, n, nref, ncols, V.as<T>());
    NSG_CUDA(cudaMemsetAsync(taup.p, 0, eb * ncols, c->stream));
    NSG_CUDA(cudaMemcpyAsync(taup.p, tau_dev, eb * nref, cudaMemcpyDeviceToDevice, c->stream));
    count_launch(c);
  }
  // S_b = V_b^H V_b over all n rows (rows above a block's reflectors are zero)
  GemmArgs g;
  g.dtype = dtype;
  g.M = NB;
  g.N = NB;
  g.K = n;
  g.A = V.p;
  g.lda = n;
  g.opA = OP_C;
  g.strideA = (int64_t)n * NB;
  g.B = V.p;
  g.ldb = n;
  g.opB = OP_N;
  g.strideB = (int64_t)n * NB;
  g.C = S.p;
  g.ldc = NB;
  g.strideC = (int64_t)NB * NB;
  g.batch = nblk;
  gemm_f64_simt(c, g);
  {
    const int shm = int(2 * NB * (NB + 1) * eb);
    raise_smem_limit((const void*)wy_tfactor_kernel<T>, shm);
    wy_tfactor_kernel<T><<<nblk, kWYThreads, shm, c->stream>>>(S.as<T>(), taup.as<T>(), Tm.as<T>());
  }
  count_launch(c);
  check_launch("back_transform factors");
}

template <typename T>
void BackTransform<T>::apply(T* Z, int64_t ldz, int64_t k) {
  if (nref == 0 || k == 0) return;
  DevBuf Wt(c, sizeof(T) * (size_t)NB * k), W2(c, sizeof(T) * (size_t)NB * k);
  for (int b = nblk - 1; b >= 0; --b) {
    const int k0 = b * NB, nbk = std::min(NB, nref - k0), rows = n - (k0 + 1);
    const T* Vb = V.as<T>() + (k0 + 1) + (size_t)k0 * n;
    // W = V_b^H Z(rows k0+1..)  (nbk x k)
    GemmArgs h;
    h.dtype = dtype;
    h.batch = 1;
    h.strideA = h.strideB = h.strideC = 0;
    h.M = nbk;
    h.N = k;
    h.K = rows;
    h.A = Vb;
    h.lda = n;
    h.opA = OP_C;
    h.B = Z + (k0 + 1);
    h.ldb = ldz;
    h.opB = OP_N;
    h.C = Wt.p;
    h.ldc = nbk;
    gemm_accurate(c, h);
    // W2 = T_b W
    GemmArgs t2 = h;
    t2.M = nbk;
    t2.N = k;
    t2.K = nbk;
    t2.A = Tm.as<T>() + (size_t)b * NB * NB;
    t2.lda = NB;
    t2.opA = OP_N;
    t2.B = Wt.p;
    t2.ldb = nbk;
    t2.opB = OP_N;
    t2.C = W2.p;
    t2.ldc = nbk;
    gemm_f64_simt(c, t2);
    // Z -= V_b W2
    GemmArgs u = h;
    u.M = rows;
    u.N = k;
    u.K = nbk;
    u.A = Vb;
    u.lda = n;
    u.opA = OP_N;
    u.B = W2.p;
    u.ldb = nbk;
    u.opB = OP_N;
    u.C = Z + (k0 + 1);
    u.ldc = ldz;
    u.alpha_re = -1.0;
    u.beta_re = 1.0;
    gemm_accurate(c, u);
  }
  check_launch("back_transform");
}

// Cluster tridiagonalisation when the matrix fits the distributed shared memory of one
// cluster (up to 16 CTAs of ~200 KB).  The cluster size comes from the tuning table by
// order (orders above the table take the kernel over all SMs), or from the context's
// override; it is raised until the columns fit.  Returns false (nothing launched) when the
// table or the override says so or when no cluster shape fits.
template <typename T>
static bool tridiag_cluster(nsg_ctx* c, int n, T* A, double* d, double* e, T* tau, double2* phase) {
  if (n < 3 || c->tune_tri == -1) return false;
  const size_t eb = sizeof(T);
  int C = c->tune_tri;
  if (C == 0) {
    for (const auto& t : tuning::kTri)
      if (n <= t.max_order) {
        C = t.path;
        break;
      }
    if (C == 0) return false;
  }
  auto kfn = tridiag_resident_kernel<T, false>;
  static_assert(kResCols >= 111, "own columns of a CTA: order 222 on two");
  for (; C <= 16; C *= 2) {
    const size_t ncol = (size_t(n) + C - 1) / C;
    const size_t smem = (ncol * n + 6 * size_t(n)) * eb;
    if (smem - 2 * size_t(n) * eb > 200 * 1024) continue;
    ensure_smem_limit((const void*)kfn, int(smem));
    if (C > 8) NSG_CUDA(cudaFuncSetAttribute((const void*)kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, (const void*)kfn, &cfg) != cudaSuccess || nclusters < 1) {
      cudaGetLastError();
      continue;
    }
    ProfScope ps(c, NSG_PROF_TRIDIAG, (sizeof(T) == 16 ? 16.0 : 4.0) / 3.0 * double(n) * n * n);
    NSG_CUDA(cudaLaunchKernelEx(&cfg, kfn, A, n, d, e, tau, phase, (ulonglong2*)nullptr, (Barrier*)nullptr));
    count_launch(c);
    check_launch("tridiag (cluster)");
    return true;
  }
  return false;
}

// The resident kernel over all SMs, when every CTA's columns fit its shared memory (real
// orders up to ~1770, complex ~1210).  Returns false with nothing launched when they do not.
template <typename T>
static bool tridiag_resident(nsg_ctx* c, int n, T* A, double* d, double* e, T* tau, double2* phase, Barrier* bar) {
  if (n < 3 || c->num_sms < 1) return false;
  const int C = std::min(c->num_sms, n);
  const size_t ncol = (size_t(n) + C - 1) / C, smem = (ncol * n + 3 * size_t(n)) * sizeof(T);
  if (ncol > size_t(kResCols) || smem > 208 * 1024) return false;
  auto kfn = tridiag_resident_kernel<T, true>;
  ensure_smem_limit((const void*)kfn, int(smem));
  int per_sm = 0;
  NSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, kResThreads, smem));
  if (per_sm < 1) return false;
  const size_t xbytes = sizeof(ulonglong2) * 4 * size_t(n) * (sizeof(T) / sizeof(double));
  DevBuf xch(c, xbytes);
  NSG_CUDA(cudaMemsetAsync(xch.p, 0, xbytes, c->stream));
  ulonglong2* px = xch.as<ulonglong2>();
  void* args[] = {&A, &n, &d, &e, &tau, &phase, &px, &bar};
  ProfScope ps(c, NSG_PROF_TRIDIAG, (sizeof(T) == 16 ? 16.0 : 4.0) / 3.0 * double(n) * n * n);
  NSG_CUDA(cudaLaunchCooperativeKernel((void*)kfn, dim3(C), dim3(kResThreads), args, smem, c->stream));
  count_launch(c);
  check_launch("tridiag (resident)");
  return true;
}

// Hermitian eigen-decomposition of A (n x n, consumed).  Eigenvalues ascending into
// w_host; eigenvectors for the eigenvalue indices `cols` (ascending order indices)
// into Zout (n x ncols, column-major).  The caller chooses cols after seeing the
// spectrum through `pick`.
template <typename T>
static void syevd_dc_impl(nsg_ctx* c, int dtype, int n, T* A, std::vector<double>& w_host, const PickFn& pick) {
  const size_t eb = sizeof(T);
  // what the host reads back, in one copy: the eigenvalues, then the leaves' error flag and
  // the grid barrier
  struct Status {
    int leaf_err, pad;
    Barrier bar;
  };
  const size_t out_bytes = sizeof(double) * n + sizeof(Status);
  DevBuf out(c, out_bytes), dd(c, sizeof(double) * n), de(c, sizeof(double) * n), dtau(c, eb * n), ph(c, sizeof(double2)),
      Q0(c, sizeof(double) * (size_t)n * n), Q1(c, sizeof(double) * (size_t)n * n);
  double* w = out.as<double>();
  Status* st = (Status*)(w + n);
  NSG_CUDA(cudaMemsetAsync(st, 0, sizeof(Status), c->stream));
  NSG_CUDA(cudaMemsetAsync(dtau.p, 0, eb * n, c->stream));
  NSG_CUDA(cudaMemsetAsync(ph.p, 0, sizeof(double2), c->stream));
  double* pd = dd.as<double>();
  double* pe = de.as<double>();
  T* pt = dtau.as<T>();
  double2* pph = ph.as<double2>();
  if (n == 1) {
    NSG_CUDA(cudaMemcpyAsync(pd, A, sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
    const double2 one = make_double2(1.0, 0.0);
    NSG_CUDA(cudaMemcpyAsync(pph, &one, sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    NSG_CUDA(cudaStreamSynchronize(c->stream));  // `one` leaves scope
  } else if (!tridiag_cluster<T>(c, n, A, pd, pe, pt, pph) && !tridiag_resident<T>(c, n, A, pd, pe, pt, pph, &st->bar)) {
    // cooperative tridiagonalisation, the matrix in L2
    int max_blocks = 0;
    size_t shm = eb * 3 * n;
    NSG_CHECK(shm <= 200 * 1024, NSG_ERR_UNSUPPORTED, "tridiagonalisation: matrix order too large");
    // one CTA per SM: the active CTAs (the first nact block indices) are then spread over
    // all SMs.  256 threads (two warps per SM sub-partition) for real data, 128 for complex
    // data (measured: 128 threads 17 % slower for real, 6 % faster for complex at n = 1024;
    // 512 threads and two CTAs per SM slower for both)
    constexpr int kTriThreads = sizeof(T) == 8 ? 256 : 128;
    auto kfn = tridiag_kernel<T, kTriThreads>;
    raise_smem_limit((const void*)kfn, int(shm));
    NSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_blocks, kfn, kTriThreads, shm));
    NSG_CHECK(max_blocks > 0, NSG_ERR_UNSUPPORTED, "tridiagonalisation: no resident block fits");
    int64_t want = ((int64_t)n * n + kTriThreads * 8 - 1) / (kTriThreads * 8);
    int grid = int(std::min<int64_t>({(int64_t)max_blocks * c->num_sms, std::max<int64_t>(want, 1),
                                      (int64_t)c->num_sms}));
    {
      const int64_t rb = sizeof(T) == 8 ? 512 : 256, m = n - 1;
      const int64_t units = ((m + grid - 1) / grid) * ((m + rb - 1) / rb);
      NSG_CHECK(units <= kTriUnits, NSG_ERR_UNSUPPORTED, "tridiagonalisation: matrix order too large for the grid");
    }
    DevBuf xbuf(c, eb * 2 * n), part(c, sizeof(double2) * 2 * grid);
    T* px = xbuf.as<T>();
    T* pp = part.as<T>();
    Barrier* pb = &st->bar;
    int pt_arg = 1024 / kTriThreads;  // trailing elements per thread before another CTA joins the pass
    void* args[] = {&A, &n, &pd, &pe, &pt, &px, &pp, &pb, &pt_arg, &pph};
    ProfScope ps(c, NSG_PROF_TRIDIAG, (sizeof(T) == 16 ? 16.0 : 4.0) / 3.0 * double(n) * n * n);
    NSG_CUDA(cudaLaunchCooperativeKernel((void*)kfn, dim3(grid), dim3(kTriThreads), args, shm,
                                         c->stream));
    count_launch(c);
    check_launch("tridiag");
  }
  const double* Q = tridiag_dc(c, n, pd, pe, Q0.as<double>(), Q1.as<double>(), w, &st->leaf_err);
  double* host = host_scalars(c, out_bytes / sizeof(double) + 1);
  NSG_CUDA(cudaMemcpyAsync(host, out.p, out_bytes, cudaMemcpyDeviceToHost, c->stream));
  NSG_CUDA(cudaEventRecord(read_event(c), c->stream));
  BackTransform<T> back(c, dtype, n, A, pt);  // (its factors are formed while the host reads)
  NSG_CUDA(cudaEventSynchronize(read_event(c)));
  Status hs;
  std::memcpy(&hs, host + n, sizeof(Status));
  NSG_CHECK(hs.bar.err == 0, NSG_ERR_TIMEOUT, "tridiagonalisation: grid barrier timed out");
  NSG_CHECK(hs.leaf_err == 0, NSG_ERR_NONFINITE, "eigensolver: a tridiagonal leaf or a secular root did not converge");
  w_host.assign(host, host + n);
  for (double x : w_host) NSG_CHECK(std::isfinite(x), NSG_ERR_NONFINITE, "eigensolver: non-finite eigenvalue");
  void* Zv = nullptr;
  int64_t ldz = 0;
  const EigCols cols = pick(w_host, &Zv, &ldz);
  T* Zout = (T*)Zv;
  if (cols.count == 0) return;
  const int gblocks = int(std::min<int64_t>(((int64_t)n * cols.count + 255) / 256, (int64_t)c->num_sms * 8));
  gather_vectors_kernel<<<gblocks, 256, 0, c->stream>>>(Q, n, cols.first, cols.step, cols.count, Zout, ldz, pph);
  count_launch(c);
  check_launch("eigenvector gather");
  back.apply(Zout, ldz, cols.count);
}

void syevd_dc(nsg_ctx* c, int dtype, int n, void* A, std::vector<double>& w_host, const PickFn& pick) {
  if (dtype == NSG_C128)
    syevd_dc_impl<double2>(c, dtype, n, (double2*)A, w_host, pick);
  else
    syevd_dc_impl<double>(c, dtype, n, (double*)A, w_host, pick);
}

}  // namespace nsg
