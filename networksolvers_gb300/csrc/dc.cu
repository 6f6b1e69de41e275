// Divide and conquer for the symmetric tridiagonal eigenproblem of the truncated
// factorizations (Cuppen's method: J. J. M. Cuppen, Numer. Math. 36 (1981), with the
// deflation of J. J. Dongarra and D. C. Sorensen, SIAM J. Sci. Stat. Comput. 8 (1987), and
// the recomputed weights of M. Gu and S. C. Eisenstat, SIAM J. Matrix Anal. Appl. 15
// (1994)): leaves of 8 rows (by default) diagonalised by cyclic Jacobi rotations, then a
// rank-one merge per node of a binary tree, one tree level at a time.
//
// A tree node is named by (depth, index): its rows follow from halving [0, n), so nothing
// about the tree is uploaded, and the deflation counts stay on the device (the kernels
// read them; only a level whose merge product goes to the tensor cores needs them on the
// host, and that read waits while the level's other kernels run).  The steps of a merge
// are device functions over a group of warps or CTAs, run in two forms:
//  * orders up to kFusedMax: one thread-block cluster runs the whole tree, its CTAs
//    meeting at the hardware cluster barrier between steps (one launch; merges on 16 SMs);
//  * larger orders: a launch per step and level over the whole GPU.
//
// FP64 is the scarce unit (two operations per clock and SM, 64 clocks per warp-wide
// instruction), so: reciprocals come from an FP32 seed and one third-order Newton step
// (3 FP64 operations instead of a division's ~9), the secular sums carry rho z_j^2 per
// pole, comparisons are integer ones where they can be, and the merge products skip the
// rows and columns that the two halves' block structure makes zero.
#include "nsg_internal.h"
#include "secular.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

namespace nsg {

namespace {

constexpr int kLeafMax = 32;
constexpr int kNT = 256, kNW = kNT / 32;
constexpr int kSmemMerge = 4096;  // rows of a block whose merge preparation runs in shared memory
constexpr int kPrepBytes = 40;    // shared memory per row of that preparation

// Workspace: arrays of length n, a merge of the rows [lo, hi) using the slice [lo, hi):
//   Ds, zs     sorted (sign-flipped) poles and normalised weights z
//   perm       block-local column of sorted slot t
//   kind       0 deflated, 1 kept, 3 kept and its column rotated with another
//   Dk, zk, wk the kept poles, their weights z and rho z^2, compacted
//   qcol       block-local column of the q-th kept pole
//   l1, l2     kept poles whose column has entries in the first / second half's rows
//   lam, zh    secular roots and recomputed weights
//   outp       output column of root s (s < k) or of deflated pole s - k
//   dcol       block-local column of deflated pole j
//   rot_pq, rot_cs   deflation rotations (2 entries each, at 2 lo)
//   gscr       scratch of blocks above kSmemMerge rows
//   low        exponent below which an entry of T counts as zero
// Delta and St hold nb^2 entries per merge at offset mi nbmax^2.
enum { C_K = 0, C_ROT, C_FLIP, C_L1, C_L2, C_STRIDE = 8 };
struct DcWork {
  int n, leaf;
  const double *d, *e;
  double *w, *Ds, *zs, *Dk, *zk, *wk, *lam, *zh, *rot_cs, *gscr, *rho, *Delta, *St;
  int *perm, *kind, *qcol, *l1, *l2, *outp, *dcol, *rot_pq, *counts, *low, *err;
};

struct Span {
  int lo, hi;
};
__host__ __device__ inline Span node_at(int n, int depth, int idx) {
  Span s{0, n};
  for (int b = depth - 1; b >= 0; --b) {
    const int mid = s.lo + (s.hi - s.lo) / 2;
    if ((idx >> b) & 1)
      s.lo = mid;
    else
      s.hi = mid;
  }
  return s;
}

// FP32 seeds of 1 / d and 1 / sqrt(d) (d > 0) to 2^-21, for normal d away from the ends of
// the exponent range: the function of the leading 24 significand bits in FP32, its exponent
// rebuilt by integer arithmetic.
__device__ __forceinline__ bool seed_range(double d) {
  const int e = (__double2hiint(d) >> 20) & 0x7ff;
  return e >= 64 && e <= 1982;
}
__device__ __forceinline__ double recip_seed(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(__uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29))));
  const unsigned b = __float_as_uint(f), e = (hi >> 20) & 0x7ff;
  return __hiloint2double(int((hi & 0x80000000u) | (((b >> 23) - 127 + 2046 - e) << 20) | ((b >> 3) & 0xfffffu)),
                          int(b << 29));
}
__device__ __forceinline__ double rsqrt_seed(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), e = (hi >> 20) & 0x7ff;
  // d = m 2^(2 h), m in [1, 4)
  const unsigned odd = (e + 1) & 1, h = (e - 1023 - odd);
  float f;
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(f)
      : "f"(__uint_as_float(0x3f800000u + (odd << 23) + (((hi & 0xfffffu) << 3) | (lo >> 29)))));
  const unsigned b = __float_as_uint(f);
  return __hiloint2double(int((((b >> 23) - 127 + 1023 - unsigned(int(h) >> 1)) << 20) | ((b >> 3) & 0xfffffu)),
                          int(b << 29));
}
// 1 / d to about an ulp: one third-order Newton step y + y (r + r^2), r = 1 - d y.  Numbers
// out of the seed's range (zeros and non-finite ones among them) take the division.
__device__ __forceinline__ double recip(double d) {
  if (!seed_range(d)) return 1.0 / d;
  const double y = recip_seed(d), r = fma(-d, y, 1.0);
  return fma(y, fma(r, r, r), y);
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Exclusive prefix sum of v over the CTA's threads in thread order; the total goes to
// *tot.  Every thread must call it.
__device__ int block_scan_excl(int v, int* tot) {
  __shared__ int sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int t = lane < nw ? sh[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) sh[lane] = t;
  }
  __syncthreads();
  const int before = warp > 0 ? sh[warp - 1] : 0;
  *tot = sh[nw - 1];
  __syncthreads();
  return before + x - v;
}

// Number of indices i in [0, len) with key(i) < k (strict) or key(i) <= k, for keys
// ascending in i.
template <bool kStrict, typename F>
__device__ __forceinline__ int rank_in(F key, int len, long long k) {
  int lo = 0, hi = len;
  while (lo < hi) {
    const int md = (lo + hi) >> 1;
    const long long v = key(md);
    if (kStrict ? (v < k) : (v <= k))
      lo = md + 1;
    else
      hi = md;
  }
  return lo;
}

// x, or 0 when its biased exponent is below `low`: a matrix of low rank leaves blocks of T that
// fall by eps from row to row, and the merges square their entries' differences.
__device__ __forceinline__ double above(double x, int low) {
  return ((__double2hiint(x) >> 20) & 0x7ff) < low ? 0.0 : x;
}

// One leaf (rows [lo, hi), at most 32) by one CTA: two-sided cyclic Jacobi with the
// round-robin ordering, half the rows' pairs rotated at once; a step is one pass over the
// rows of independent 2 x 2 blocks plus the eigenvector columns.  The rotation's tangent is
// chosen in FP32 (it need only come close to annihilating the pair: what it leaves is
// 2^-22 of it, and the next sweep's), its cosine and sine are orthonormal in FP64.  The
// leaf is scaled to norm about 1 by a power of two; off-diagonal entries below eps / 4 of
// that count as zero.  A rotation of two equal diagonal entries leaves rounding of that size, and
// a leaf of equal ones (of an orthogonal matrix's Gram matrix) may go on exchanging it: from the
// tenth sweep on, which few other leaves reach, the bound doubles every other sweep (at most 16
// sweeps, four eps, over three million random leaves, a ninth of them equal entries and noise).
// Measured: 48 us for leaves of 8 rows (an implicit-QL chase, a serial chain of square roots and
// divisions, 148).  Writes the sorted pairs into the leaf's diagonal block of Q0 and Q1 and into
// w; a leaf that still rotates after 30 sweeps raises *err.
__device__ void solve_leaf(const DcWork& W, int lo, int hi, double* Q0, double* Q1) {
  __shared__ double A[kLeafMax][kLeafMax + 1], V[kLeafMax][kLeafMax + 1], cs[kLeafMax / 2], sn[kLeafMax / 2];
  __shared__ int pos[kLeafMax], moved, expo, top;
  __shared__ unsigned char pairs[kLeafMax - 1][kLeafMax / 2][2];  // of round r: (lower, upper) index
  const int s = hi - lo, tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) {
    moved = 0;
    expo = 0;
    top = 0;
  }
  __syncthreads();
  // entries below 2^-200 of T's largest count as zero (the same bound in every CTA)
  int mx = 0;
  for (int i = tid; i < W.n; i += nt)
    mx = max(mx, max((__double2hiint(W.d[i]) >> 20) & 0x7ff, i + 1 < W.n ? (__double2hiint(W.e[i]) >> 20) & 0x7ff : 0));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0) atomicMax(&top, mx);
  __syncthreads();
  const int low = max(top - 200, 0);
  if (tid == 0) *W.low = low;
  for (int t = tid; t < s * s; t += nt) {
    const int i = t % s, j = t / s;
    double a = 0.0;
    if (i == j) {  // the rank-one updates of the splits at both ends are taken off
      a = above(W.d[lo + i], low);
      if (i == 0 && lo > 0) a -= above(W.e[lo - 1], low);
      if (i == s - 1 && hi < W.n) a -= above(W.e[hi - 1], low);
    } else if (i == j + 1 || j == i + 1) {
      a = above(W.e[lo + min(i, j)], low);
    }
    A[i][j] = a;
    V[i][j] = i == j ? 1.0 : 0.0;
    atomicMax(&expo, (__double2hiint(a) >> 20) & 0x7ff);
  }
  __syncthreads();
  // (a leaf near the ends of the exponent range or not finite keeps a smaller scale; a zero
  // leaf rotates nothing)
  const int shift = 1023 - min(max(expo, 64), 1982);
  const double up = __hiloint2double((1023 + shift) << 20, 0), down = __hiloint2double((1023 - shift) << 20, 0);
  for (int t = tid; t < s * s; t += nt) A[t % s][t / s] *= up;
  const int ne = s + (s & 1), np = ne / 2;  // an odd order has a bye (index s)
  for (int t = tid; t < (ne - 1) * np; t += nt) {
    const int r = t / np, m = t % np;
    const int x = m == 0 ? ne - 1 : (r + m) % (ne - 1), y = m == 0 ? r : (r - m + ne - 1) % (ne - 1);
    pairs[r][m][0] = (unsigned char)min(x, y);
    pairs[r][m][1] = (unsigned char)max(x, y);
  }
  // a thread's items of every step: row h of the 2 x 2 block of pairs (a, b), the two rows of
  // a block on neighbouring lanes; then row i of the eigenvector columns of pair m
  const int nblk = 2 * np * np, vbase = (nblk + 31) & ~31, nitems = vbase + np * s;
  int ia[4], ib[4];
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const int t = tid + x * nt;
    ia[x] = t < vbase ? (t >> 1) % np : (t - vbase) / s;
    ib[x] = t < vbase ? (t >> 1) / np : (t - vbase) % s;
  }
  __syncthreads();
  float tiny = 1.2e-16f;
  for (int sweep = 0; s > 1; ++sweep) {
    for (int r = 0; r < ne - 1; ++r) {
      if (tid < np) {
        const int p = pairs[r][tid][0], q = pairs[r][tid][1];
        double c = 1.0, sv = 0.0;
        if (q < s) {
          const float h = 2.0f * (float)A[p][q];
          if (fabsf(h) > tiny) {
            const float d = (float)(A[q][q] - A[p][p]);
            const float t = h / (fabsf(d) + sqrtf(fmaf(d, d, h * h)));
            const double tt = (double)copysignf(t, h * copysignf(1.0f, d));
            const double g = fma(tt, tt, 1.0), y = rsqrt_seed(g);  // g in [1, 2]
            const double e = fma(-g * y, y, 1.0);
            c = fma(y * e, fma(0.375, e, 0.5), y);
            sv = tt * c;
            moved = 1;
          }
        }
        cs[tid] = c;
        sn[tid] = sv;
      }
      __syncthreads();
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int t = tid + x * nt;
        if (t >= nitems) break;  // (whole warps below vbase)
        if (t < vbase) {
          const int a = ia[x], b = ib[x], h = t & 1;
          double u0 = 0.0, v0 = 0.0;
          int row = 0, u = 0, v = 0;
          bool act = false;
          if (t < nblk && (sn[a] != 0.0 || sn[b] != 0.0)) {
            row = pairs[r][a][h];
            const int other = pairs[r][a][1 - h];
            u = pairs[r][b][0];
            v = pairs[r][b][1];
            act = row < s;
            if (act) {  // (a bye's partner index is s: its rotation is the identity)
              const double ca = cs[a], sa = h ? sn[a] : -sn[a], cb = cs[b], sb = sn[b];
              const double x0 = A[row][u], x1 = v < s ? A[row][v] : 0.0;
              const double y0 = other < s ? A[other][u] : 0.0, y1 = other < s && v < s ? A[other][v] : 0.0;
              const double r0 = fma(sa, y0, ca * x0), r1 = fma(sa, y1, ca * x1);
              u0 = fma(-sb, r1, cb * r0);
              v0 = fma(sb, r0, cb * r1);
            }
          }
          __syncwarp();  // both rows of a block are read before either is written
          if (act) {
            A[row][u] = u0;
            if (v < s) A[row][v] = v0;
          }
        } else {
          const int m = ia[x], i = ib[x], p = pairs[r][m][0], q = pairs[r][m][1];
          if (q < s && sn[m] != 0.0) {
            const double vx = V[i][p], vy = V[i][q];
            V[i][p] = fma(-sn[m], vy, cs[m] * vx);
            V[i][q] = fma(sn[m], vx, cs[m] * vy);
          }
        }
      }
      __syncthreads();
    }
    const int any = moved;
    __syncthreads();
    if (tid == 0) moved = 0;
    __syncthreads();
    if (!any) break;
    if (sweep == 30) {
      if (tid == 0) atomicExch(W.err, 1);
      break;
    }
    if (sweep >= 9 && (sweep & 1)) tiny *= 2.f;
  }
  if (tid < s) {
    const long long k = order_key(A[tid][tid]);
    int r = 0;
    for (int j = 0; j < s; ++j) {
      const long long kj = order_key(A[j][j]);
      r += kj < k || (kj == k && j < tid);
    }
    pos[tid] = r;
    W.w[lo + r] = A[tid][tid] * down;
  }
  __syncthreads();
  for (int t = tid; t < s * s; t += nt) {
    const int i = t % s, j = t / s;
    const size_t o = (size_t)(lo + pos[j]) * W.n + (lo + i);
    Q0[o] = V[i][j];
    Q1[o] = V[i][j];
  }
  __syncthreads();
}

// Preparation of one merge by one CTA: gather the halves' eigenvalues and the z vector
// (last row of the first half, first row of the second), flip for rho < 0, merge the
// ascending halves, normalise z, deflate (small weights; poles closer than the tolerance
// rotated together) and compact the kept poles.
__device__ void prep_merge(const DcWork& W, const double* Q, int lo, int hi, int mi, double* smem) {
  const int n = W.n, nb = hi - lo, n1 = nb / 2, n2 = nb - n1, mid = lo + n1, tid = threadIdx.x, nt = blockDim.x;
  const bool sm = nb <= kSmemMerge;
  double* ws = sm ? smem : W.gscr + 2 * (size_t)lo;  // block eigenvalues by local index
  double* zr = ws + nb;                              // z candidates by local index
  double* Dsm = sm ? zr + nb : W.Ds + lo;
  double* zsm = sm ? Dsm + nb : W.zs + lo;
  int* pm = sm ? (int*)(zsm + nb) : W.perm + lo;
  int* kd = sm ? pm + nb : W.kind + lo;
  __shared__ double red[kNW];
  __shared__ long long redm[kNW];
  __shared__ double s_nz, s_dmax;
  __shared__ int s_flag, s_nrot;
  for (int li = tid; li < nb; li += nt) {
    ws[li] = W.w[lo + li];
    zr[li] = Q[(size_t)(lo + li) * n + (li < n1 ? mid - 1 : mid)];
  }
  if (tid == 0) {
    s_flag = 0;
    s_nrot = 0;
  }
  __syncthreads();
  double rho = above(W.e[mid - 1], *W.low);
  const int flip = rho < 0;
  if (flip) rho = -rho;
  // merge of the two ascending halves (both traversed from their top when flipped, values
  // negated) into ascending poles; ties take the first half first.  An entry's slot is
  // its rank in its own half plus its rank in the other, by binary search on integer keys.
  auto srcA = [&](int a) { return flip ? (n1 - 1 - a) : a; };
  auto srcB = [&](int b) { return flip ? (nb - 1 - b) : (n1 + b); };
  auto keyA = [&](int a) { return order_key(flip ? neg_exact(ws[srcA(a)]) : ws[srcA(a)]); };
  auto keyB = [&](int b) { return order_key(flip ? neg_exact(ws[srcB(b)]) : ws[srcB(b)]); };
  for (int t = tid; t < nb; t += nt)  // halves out of order: the serial merge
    if ((t > 0 && t < n1 && keyA(t) < keyA(t - 1)) || (t > n1 && keyB(t - n1) < keyB(t - n1 - 1))) s_flag = 1;
  __syncthreads();
  auto place = [&](int slot, int li) {
    pm[slot] = li;
    Dsm[slot] = flip ? neg_exact(ws[li]) : ws[li];
    zsm[slot] = zr[li];
  };
  if (!s_flag) {
    for (int t = tid; t < nb; t += nt) {
      if (t < n1)
        place(t + rank_in<true>(keyB, n2, keyA(t)), srcA(t));
      else
        place((t - n1) + rank_in<false>(keyA, n1, keyB(t - n1)), srcB(t - n1));
    }
  } else if (tid == 0) {
    int a = 0, b = 0;
    for (int t = 0; t < nb; ++t) {
      const bool takeA = a < n1 && (b >= n2 || keyA(a) <= keyB(b));
      place(t, takeA ? srcA(a) : srcB(b));
      if (takeA)
        ++a;
      else
        ++b;
    }
  }
  __syncthreads();
  // |z| and max |D| (fixed-order block reductions; the largest magnitude by its bits)
  double s2 = 0.0;
  long long dm = 0;
  for (int t = tid; t < nb; t += nt) {
    s2 = fma(zsm[t], zsm[t], s2);
    dm = max(dm, __double_as_longlong(Dsm[t]) & 0x7fffffffffffffffLL);
  }
  s2 = warp_sum(s2);
  for (int o = 16; o > 0; o >>= 1) dm = max(dm, __shfl_xor_sync(0xffffffffu, dm, o));
  const int warp = tid >> 5, lane = tid & 31;
  if (lane == 0) {
    red[warp] = s2;
    redm[warp] = dm;
  }
  __syncthreads();
  if (warp == 0) {
    double v = lane < kNW ? red[lane] : 0.0;
    long long m = lane < kNW ? redm[lane] : 0;
    for (int o = kNW / 2; o > 0; o >>= 1) {
      v += __shfl_xor_sync(0xffffffffu, v, o);
      m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    if (lane == 0) {
      s_nz = sqrt(v);
      s_dmax = __longlong_as_double(m);
      s_flag = 0;
    }
  }
  __syncthreads();
  const double nz = s_nz, inz = 1.0 / nz;
  rho = rho * nz * nz;
  const double tol = 8.0 * kEps * fmax(s_dmax, rho);
  // deflation of small weights (independent per pole), then of poles closer than tol:
  // the closest pairs of kept poles are neighbours among the kept ones
  for (int t = tid; t < nb; t += nt) {
    const double z = zsm[t] * inz;
    const bool small = rho * fabs(z) <= tol;
    kd[t] = small ? 0 : 1;
    zsm[t] = small ? 0.0 : z;
  }
  __syncthreads();
  for (int t = tid; t < nb; t += nt) {
    if (!kd[t]) continue;
    for (int u = t + 1; u < nb; ++u)
      if (kd[u]) {
        if (fabs(Dsm[u] - Dsm[t]) <= tol) s_flag = 1;
        break;
      }
  }
  __syncthreads();
  const int per = (nb + nt - 1) / nt, c0 = min(nb, tid * per), c1 = min(nb, c0 + per);
  if (s_flag) {
    // the rotation sweep: serial along runs of close neighbours only.  Kept slots ks, and
    // the kept indices a whose neighbour a + 1 is close (in ws and zr, no longer needed).
    int* ks = (int*)ws;
    int* fl = (int*)zr;
    int cnt = 0, kept = 0, nfl = 0;
    for (int t = c0; t < c1; ++t) cnt += kd[t] != 0;
    int off = block_scan_excl(cnt, &kept);
    for (int t = c0; t < c1; ++t)
      if (kd[t]) ks[off++] = t;
    __syncthreads();
    const int pk = (kept + nt - 1) / nt, a0 = min(kept, tid * pk), a1 = min(kept, a0 + pk);
    auto close = [&](int a) { return a + 1 < kept && fabs(Dsm[ks[a + 1]] - Dsm[ks[a]]) <= tol; };
    cnt = 0;
    for (int a = a0; a < a1; ++a) cnt += close(a);
    off = block_scan_excl(cnt, &nfl);
    for (int a = a0; a < a1; ++a)
      if (close(a)) fl[off++] = a;
    __syncthreads();
    if (tid == 0) {
      int* rpq = W.rot_pq + 2 * lo;
      double* rcs = W.rot_cs + 2 * lo;
      int nrot = 0, done = 0;
      for (int f = 0; f < nfl; ++f) {
        if (fl[f] < done) continue;
        int a = fl[f];
        while (close(a)) {
          const int prev = ks[a], t = ks[a + 1];
          const double r = hypot(zsm[t], zsm[prev]);
          const double c = zsm[t] / r, sn = zsm[prev] / r;
          const double dp = Dsm[prev], dt = Dsm[t];
          Dsm[prev] = c * c * dp + sn * sn * dt;
          Dsm[t] = sn * sn * dp + c * c * dt;
          zsm[prev] = 0.0;
          zsm[t] = r;
          kd[prev] = 0;
          kd[t] = 3;
          rpq[2 * nrot] = pm[prev];
          rpq[2 * nrot + 1] = pm[t];
          rcs[2 * nrot] = c;
          rcs[2 * nrot + 1] = sn;
          ++nrot;
          ++a;
        }
        done = a;
      }
      s_nrot = nrot;
    }
    __syncthreads();
  }
  // compaction of the kept slots, and of those with entries in either half's rows
  int cnt = 0, both = 0;
  auto in1 = [&](int t) { return kd[t] == 3 || pm[t] < n1; };
  auto in2 = [&](int t) { return kd[t] == 3 || pm[t] >= n1; };
  for (int t = c0; t < c1; ++t)
    if (kd[t]) {
      ++cnt;
      both += (in1(t) ? 1 : 0) + (in2(t) ? 1 << 16 : 0);
    }
  int k = 0, tot = 0;
  int off = block_scan_excl(cnt, &k);
  const int offs = block_scan_excl(both, &tot);
  int o1 = offs & 0xffff, o2 = offs >> 16;
  for (int t = c0; t < c1; ++t)
    if (kd[t]) {
      W.qcol[lo + off] = pm[t];
      W.Dk[lo + off] = Dsm[t];
      W.zk[lo + off] = zsm[t];
      W.wk[lo + off] = rho * zsm[t] * zsm[t];
      if (in1(t)) W.l1[lo + o1++] = off;
      if (in2(t)) W.l2[lo + o2++] = off;
      ++off;
    }
  if (tid == 0) {
    W.rho[mi] = rho;
    int* ct = W.counts + C_STRIDE * mi;
    ct[C_K] = k;
    ct[C_ROT] = s_nrot;
    ct[C_FLIP] = flip;
    ct[C_L1] = tot & 0xffff;
    ct[C_L2] = tot >> 16;
  }
  if (sm)
    for (int t = tid; t < nb; t += nt) {
      W.Ds[lo + t] = Dsm[t];
      W.perm[lo + t] = pm[t];
      W.kind[lo + t] = kd[t];
    }
  __syncthreads();
}

// One secular root (secular.h) by a group of G lanes (the 32 / G groups of a warp work on as
// many roots, so the scalar part of a step, most of it at small k, serves them all).  Groups
// without a root (i >= k) and finished ones keep their warp company.
template <int G>
__device__ void secular_root(const DcWork& W, int lo, int k, int i, double rho, int lane, double* Delta) {
  const double* Dk = W.Dk + lo;
  const double* wk = W.wk + lo;
  const int gl = lane & (G - 1);
  const bool real = i < k;
  if (!real) i = 0;
  constexpr int RC = 8;  // poles per lane held in registers
  double dj[RC], wr[RC], dd[RC];
#pragma unroll
  for (int t = 0; t < RC; ++t) {
    const int j = gl + G * t;
    dj[t] = j < k ? Dk[j] : 0.0;
    wr[t] = j < k ? wk[j] : 0.0;
  }
  const double Di = k > 0 ? Dk[i] : 0.0, gap = i < k - 1 ? Dk[i + 1] - Di : 0.0;
  double dorg = Di;
  auto recenter = [&]() {
#pragma unroll
    for (int t = 0; t < RC; ++t)
      if (G * t < k) dd[t] = dj[t] - dorg;
  };
  recenter();
  double f, dr;  // the secular function and its slope at tau without pole `skip`'s part
  float fa;      // the sum of its terms' magnitudes
  auto eval = [&](double tau, int skip) {
    double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;  // poles j <= i (terms <= 0), j > i (>= 0)
    auto term = [&](int j, double del, double w) {
      const double r = recip(del), a = w * r, b = j == skip ? 0.0 : a * r;
      if (j <= i) {
        psi += a;
        dpsi += b;
      } else {
        phi += a;
        dphi += b;
      }
    };
#pragma unroll
    for (int t = 0; t < RC; ++t) {
      const int j = gl + G * t;
      if (j < k) term(j, dd[t] - tau, wr[t]);
    }
    for (int j = gl + G * RC; j < k; j += G) term(j, (Dk[j] - dorg) - tau, wk[j]);
    // the four sums over the group with log2(G) + 1 additions: the first two steps fold the
    // lanes of one value into half the lanes of another
    const bool h1 = lane & (G / 2), h2 = lane & (G / 4);
    double x = h1 ? phi : psi, y = h1 ? dphi : dpsi;
    x += __shfl_xor_sync(0xffffffffu, h1 ? psi : phi, G / 2);
    y += __shfl_xor_sync(0xffffffffu, h1 ? dpsi : dphi, G / 2);
    double v = h2 ? y : x;
    v += __shfl_xor_sync(0xffffffffu, h2 ? x : y, G / 4);
#pragma unroll
    for (int o = G / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    // the group's lane 0 holds psi, G / 4 dpsi, G / 2 phi, 3 G / 4 dphi
    const double o2 = __shfl_xor_sync(0xffffffffu, v, G / 2), sum = v + o2;
    f = 1.0 + __shfl_sync(0xffffffffu, sum, 0, G);
    dr = __shfl_sync(0xffffffffu, sum, G / 4, G);
    fa = __shfl_sync(0xffffffffu, fabsf((float)v - (float)o2), 0, G);
  };
  const bool inner = i < k - 1;
  double blo = 0.0, bhi = inner ? gap : rho, tau = 0.5 * bhi, ddi = 0.0, ddi1 = gap;
  eval(tau, -1);
  if (inner) {
    const double mid = tau;
    if (f >= 0) {
      bhi = mid;
    } else {
      dorg = Dk[i + 1];
      recenter();
      tau = -mid;
      blo = -mid;
      bhi = 0.0;
      ddi = -gap;
      ddi1 = 0.0;
    }
  }
  SecularRoot root;
  root.dorg = dorg;
  root.tau = tau;
  root.blo = blo;
  root.bhi = bhi;
  root.ftol = float(4.0 * kEps) * float(k + 1);
  root.fprev = INFINITY;
  root.inner = inner;
  root.single = k <= 1;
  root.left = dorg == Di;
  root.q1 = inner ? ddi : (k > 1 ? Dk[k - 2] - dorg : 0.0);
  root.q2 = inner ? ddi1 : 0.0;
  root.jorg = inner && !root.left ? i + 1 : i;
  root.worg = k > 0 ? wk[root.jorg] : 0.0;
  auto reciprocal = [](double d) { return recip(d); };
  auto quotient = [](float a, float b) { return __fdividef(a, b); };
  bool done = !real;
  for (int it = 0; it < kSecularSteps; ++it) {
    if (it > 0) eval(root.tau, root.jorg);
    if (!done) done = root.step(it, f, dr, fa, reciprocal, quotient);
    if (__all_sync(0xffffffffu, done)) break;
  }
  if (!real) return;
  if (gl == 0) W.lam[lo + i] = root.dorg + root.tau;
  if (gl == 0 && !done) atomicExch(W.err, 1);
  for (int j = gl; j < k; j += G) Delta[(size_t)i * k + j] = (Dk[j] - root.dorg) - root.tau;
}

// Lanes per root: the fewest (8 at least) with which the roots' warps still do not exceed
// one per SM sub-partition.
__host__ __device__ inline int secular_lanes(int roots, int subparts) {
  int g = 32;
  while (g > 8 && roots * g > 32 * subparts) g /= 2;
  return g;
}
// roots (merge mi, index i), numbered mi nbmax + i, of a level by the warp's groups
template <int G>
__device__ void secular_group(const DcWork& W, int depth, int nbmax, int warp_item, int lane) {
  const int g = warp_item * (32 / G) + lane / G, nm = 1 << depth;
  const int mi = min(g / nbmax, nm - 1), i = g / nbmax < nm ? g % nbmax : nbmax;
  const int k = W.counts[C_STRIDE * mi + C_K];
  if (__all_sync(0xffffffffu, i >= k)) return;
  secular_root<G>(W, node_at(W.n, depth, mi).lo, k, i, W.rho[mi], lane, W.Delta + (size_t)mi * nbmax * nbmax);
}
__device__ void secular_item(const DcWork& W, int depth, int nbmax, int lanes, int warp_item, int lane) {
  if (lanes == 32)
    secular_group<32>(W, depth, nbmax, warp_item, lane);
  else if (lanes == 16)
    secular_group<16>(W, depth, nbmax, warp_item, lane);
  else
    secular_group<8>(W, depth, nbmax, warp_item, lane);
}

// Recomputed weight j of a merge by one warp:
// zhat_j^2 = (lam_j - D_j) / rho * prod_{i != j} (lam_i - D_j) / (D_i - D_j)
__device__ void gu_eisenstat(const DcWork& W, int lo, int k, int j, double rho, int lane, const double* Delta) {
  const double* Dk = W.Dk + lo;
  const double dj = Dk[j];
  double p = 1.0;
  for (int i = lane; i < k; i += 32)
    if (i != j) p *= neg_exact(Delta[(size_t)i * k + j]) * recip(Dk[i] - dj);
  for (int o = 16; o > 0; o >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, o);
  if (lane == 0) {
    p *= neg_exact(Delta[(size_t)j * k + j]) / rho;
    W.zh[lo + j] = copysign(sqrt(fmax(p, 0.0)), W.zk[lo + j]);
  }
}

// Column i of S^T (the normalised eigenvector of root i) by one warp, zeros up to `pad`.
__device__ void secular_vector(const DcWork& W, int lo, int k, int i, int lane, const double* Delta, double* St, int ld,
                               int pad) {
  double* out = St + (size_t)i * ld;
  if (i >= k) {
    for (int j = lane; j < pad; j += 32) out[j] = 0.0;
    return;
  }
  const double* zh = W.zh + lo;
  const double* De = Delta + (size_t)i * k;
  constexpr int RC = 8;
  double sr[RC], nrm = 0.0;
#pragma unroll
  for (int t = 0; t < RC; ++t) {
    const int j = lane + 32 * t;
    sr[t] = j < k ? zh[j] * recip(De[j]) : 0.0;
    if (j < k) nrm = fma(sr[t], sr[t], nrm);
  }
  for (int j = lane + 32 * RC; j < k; j += 32) {
    const double s = zh[j] * recip(De[j]);
    nrm = fma(s, s, nrm);
  }
  nrm = 1.0 / sqrt(warp_sum(nrm));
#pragma unroll
  for (int t = 0; t < RC; ++t) {
    const int j = lane + 32 * t;
    if (j < k) out[j] = sr[t] * nrm;
  }
  for (int j = lane + 32 * RC; j < k; j += 32) out[j] = zh[j] * recip(De[j]) * nrm;
  for (int j = k + lane; j < pad; j += 32) out[j] = 0.0;
}

// Final ordering of one merge by one CTA: eigenvalues = roots (kept) and deflated poles,
// signs undone, ascending; the output column of each.
__device__ void order_merge(const DcWork& W, int lo, int hi, int mi, double* smem) {
  const int nb = hi - lo, tid = threadIdx.x, nt = blockDim.x;
  const int* ct = W.counts + C_STRIDE * mi;
  const int nr = ct[C_K], flip = ct[C_FLIP], nd = nb - nr;
  const bool sm = nb <= kSmemMerge;
  double* lm = sm ? smem : W.lam + lo;       // roots
  double* dv = sm ? lm + nb : W.gscr + 2 * (size_t)lo;  // deflated poles in slot order
  __shared__ int s_unsorted;
  if (tid == 0) s_unsorted = 0;
  const int per = (nb + nt - 1) / nt, c0 = min(nb, tid * per), c1 = min(nb, c0 + per);
  int cnt = 0, tot = 0;
  for (int t = c0; t < c1; ++t) cnt += W.kind[lo + t] == 0;
  int off = block_scan_excl(cnt, &tot);
  for (int t = c0; t < c1; ++t)
    if (W.kind[lo + t] == 0) {
      dv[off] = W.Ds[lo + t];
      W.dcol[lo + off++] = W.perm[lo + t];
    }
  if (sm)
    for (int t = tid; t < nr; t += nt) lm[t] = W.lam[lo + t];
  __syncthreads();
  // a stable merge of the ascending roots with the deflated poles (ties: the root first)
  // by ranks on integer keys; poles moved by a deflation rotation can be out of order by
  // up to the deflation tolerance, and then the merge is the serial one
  auto keyR = [&](int i) { return order_key(lm[i]); };
  auto keyD = [&](int j) { return order_key(dv[j]); };
  for (int i = tid + 1; i < nr; i += nt)
    if (keyR(i) < keyR(i - 1)) s_unsorted = 1;
  for (int j = tid + 1; j < nd; j += nt)
    if (keyD(j) < keyD(j - 1)) s_unsorted = 1;
  __syncthreads();
  auto put = [&](int s, int at, double v) {
    const int out = flip ? (nb - 1 - at) : at;
    W.outp[lo + s] = out;
    W.w[lo + out] = flip ? neg_exact(v) : v;
  };
  if (!s_unsorted) {
    for (int i = tid; i < nr; i += nt) put(i, i + rank_in<true>(keyD, nd, keyR(i)), lm[i]);
    for (int j = tid; j < nd; j += nt) put(nr + j, j + rank_in<false>(keyR, nr, keyD(j)), dv[j]);
  } else if (tid == 0) {
    int ia = 0, ib = 0;
    for (int at = 0; at < nb; ++at) {
      const bool root = ia < nr && (ib >= nd || keyR(ia) <= keyD(ib));
      if (root) {
        put(ia, at, lm[ia]);
        ++ia;
      } else {
        put(nr + ib, at, dv[ib]);
        ++ib;
      }
    }
  }
  __syncthreads();
}

// The deflation rotations of a merge on row r of its block of Q, in order.
__device__ void rotate_row(const DcWork& W, double* Q, int lo, int nrot, int r) {
  const int* rpq = W.rot_pq + 2 * lo;
  const double* rcs = W.rot_cs + 2 * lo;
  double* row = Q + (lo + r);
  for (int q = 0; q < nrot; ++q) {
    const size_t cp = (size_t)(lo + rpq[2 * q]) * W.n, ci = (size_t)(lo + rpq[2 * q + 1]) * W.n;
    const double c = rcs[2 * q], sn = rcs[2 * q + 1];
    const double xp = row[cp], xi = row[ci];
    row[cp] = c * xp - sn * xi;
    row[ci] = sn * xp + c * xi;
  }
}

// Tiles of a merge product: 16 rows of one half x 16 output slots (roots, then deflated
// columns, which are copied).
constexpr int MT = 16, MK = 32;
__host__ __device__ inline int merge_row_tiles(int nb) { return (nb / 2 + MT - 1) / MT + (nb - nb / 2 + MT - 1) / MT; }
__host__ __device__ inline int merge_tiles(int nb) { return merge_row_tiles(nb) * ((nb + MT - 1) / MT); }

// One tile by one CTA of 256 threads: new eigenvector columns = (kept columns) S^T, where
// a half's rows meet only the kept columns listed for that half, written to their final
// places in Qn.
__device__ void merge_tile(const DcWork& W, const double* Q, double* Qn, int lo, int hi, int mi, int tile, const double* St,
                           int ld) {
  __shared__ double As[2][MK][MT + 1], Bs[2][MK][MT + 1];
  const int n = W.n, nb = hi - lo, n1 = nb / 2, tid = threadIdx.x, ti = tid % MT, tj = tid / MT;
  const int t1 = (n1 + MT - 1) / MT, rt = merge_row_tiles(nb);
  const int rti = tile % rt, s0 = tile / rt * MT;
  const bool first = rti < t1;
  const int r0 = first ? rti * MT : n1 + (rti - t1) * MT, rend = first ? n1 : nb;
  const int* ct = W.counts + C_STRIDE * mi;
  const int k = ct[C_K], K = s0 < k ? (first ? ct[C_L1] : ct[C_L2]) : 0;
  const int* list = (first ? W.l1 : W.l2) + lo;
  double ra[MK / MT], rb[MK / MT];
  auto load = [&](int k0) {
#pragma unroll
    for (int r = 0; r < MK / MT; ++r) {
      const int qa = k0 + tj + MT * r, qb = k0 + ti + MT * r;
      ra[r] = (r0 + ti < rend && qa < K) ? Q[(size_t)(lo + W.qcol[lo + list[qa]]) * n + (lo + r0 + ti)] : 0.0;
      rb[r] = (s0 + tj < k && qb < K) ? St[(size_t)(s0 + tj) * ld + list[qb]] : 0.0;
    }
  };
  double acc = 0.0;
  if (K > 0) load(0);
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += MK, buf ^= 1) {
#pragma unroll
    for (int r = 0; r < MK / MT; ++r) {
      As[buf][tj + MT * r][ti] = ra[r];
      Bs[buf][ti + MT * r][tj] = rb[r];
    }
    __syncthreads();
    if (k0 + MK < K) load(k0 + MK);
    const int kn = min(MK, K - k0);
    if (kn == MK) {
#pragma unroll
      for (int q = 0; q < MK; ++q) acc = fma(As[buf][q][ti], Bs[buf][q][tj], acc);
    } else {
      for (int q = 0; q < kn; ++q) acc = fma(As[buf][q][ti], Bs[buf][q][tj], acc);
    }
  }
  const int s = s0 + tj;
  if (r0 + ti < rend && s < nb) {
    const double v = s < k ? acc : Q[(size_t)(lo + W.dcol[lo + s - k]) * n + (lo + r0 + ti)];
    Qn[(size_t)(lo + W.outp[lo + s]) * n + (lo + r0 + ti)] = v;
  }
  __syncthreads();  // the slabs are read before the CTA's next tile is stored
}

// ---- a launch per step and level -------------------------------------------------
__global__ void __launch_bounds__(kNT) dc_leaf_kernel(DcWork W, int levels, double* Q0, double* Q1) {
  // leaf b of depth `levels`; a node of the depth above that is a leaf already is its
  // first child's
  const Span up = node_at(W.n, max(levels - 1, 0), blockIdx.x >> 1);
  Span s = node_at(W.n, levels, blockIdx.x);
  if (levels > 0 && up.hi - up.lo <= W.leaf) {
    if (blockIdx.x & 1) return;
    s = up;
  }
  solve_leaf(W, s.lo, s.hi, Q0, Q1);
}

__global__ void __launch_bounds__(kNT) dc_prep_kernel(DcWork W, int depth, const double* Q) {
  extern __shared__ __align__(16) double dc_smem[];
  const Span s = node_at(W.n, depth, blockIdx.x);
  if (s.hi - s.lo <= W.leaf) {
    if (threadIdx.x < C_STRIDE) W.counts[C_STRIDE * blockIdx.x + threadIdx.x] = 0;
    return;
  }
  prep_merge(W, Q, s.lo, s.hi, blockIdx.x, dc_smem);
}

__global__ void __launch_bounds__(kNT) dc_secular_kernel(DcWork W, int depth, int nbmax, int lanes) {
  secular_item(W, depth, nbmax, lanes, (blockIdx.x * kNT + threadIdx.x) >> 5, threadIdx.x & 31);
}

// the orderings (first CTAs), the deflation rotations, and the recomputed weights: all
// depend on the roots at most, and on none of each other
__global__ void __launch_bounds__(kNT) dc_weights_kernel(DcWork W, int depth, int nbmax, double* Q) {
  extern __shared__ __align__(16) double dc_smem[];
  const int nm = 1 << depth, rb = (nbmax + kNT - 1) / kNT;
  int b = blockIdx.x;
  if (b < nm) {
    const Span s = node_at(W.n, depth, b);
    if (s.hi - s.lo > W.leaf) order_merge(W, s.lo, s.hi, b, dc_smem);
    return;
  }
  b -= nm;
  if (b < nm * rb) {
    const int mi = b / rb, r = b % rb * kNT + threadIdx.x;
    const Span s = node_at(W.n, depth, mi);
    const int nrot = W.counts[C_STRIDE * mi + C_ROT];
    if (nrot > 0 && r < s.hi - s.lo) rotate_row(W, Q, s.lo, nrot, r);
    return;
  }
  b -= nm * rb;
  const int gw = (b * kNT + threadIdx.x) >> 5, mi = gw / nbmax, j = gw % nbmax;
  if (mi >= nm || j >= W.counts[C_STRIDE * mi + C_K]) return;
  gu_eisenstat(W, node_at(W.n, depth, mi).lo, W.counts[C_STRIDE * mi + C_K], j, W.rho[mi], threadIdx.x & 31,
               W.Delta + (size_t)mi * nbmax * nbmax);
}

// (pad: zero the columns and rows beyond k, for the padded batched product)
__global__ void __launch_bounds__(kNT) dc_vectors_kernel(DcWork W, int depth, int nbmax, bool pad) {
  const int gw = (blockIdx.x * kNT + threadIdx.x) >> 5, mi = gw / nbmax, i = gw % nbmax;
  if (mi >= (1 << depth)) return;
  const int k = W.counts[C_STRIDE * mi + C_K];
  if (i >= k && !pad) return;
  const size_t o = (size_t)mi * nbmax * nbmax;
  secular_vector(W, node_at(W.n, depth, mi).lo, k, i, threadIdx.x & 31, W.Delta + o, W.St + o, nbmax, pad ? nbmax : 0);
}

__global__ void __launch_bounds__(kNT) dc_merge_kernel(DcWork W, int depth, int nbmax, const double* Q, double* Qn) {
  const Span s = node_at(W.n, depth, blockIdx.y);
  if (s.hi - s.lo <= W.leaf || int(blockIdx.x) >= merge_tiles(s.hi - s.lo)) return;
  merge_tile(W, Q, Qn, s.lo, s.hi, blockIdx.y, blockIdx.x, W.St + (size_t)blockIdx.y * nbmax * nbmax, nbmax);
}

// The kept columns of each block, compacted into an nbmax x kmax matrix per merge (zero
// padded), for the batched product; blockIdx.y = merge.
__global__ void dc_gather_kernel(DcWork W, int depth, int nbmax, int kmax, const double* __restrict__ Q,
                                 double* __restrict__ Qk_all) {
  const int mi = blockIdx.y;
  const Span s = node_at(W.n, depth, mi);
  const int lo = s.lo, nb = s.hi - s.lo, k = W.counts[C_STRIDE * mi + C_K];
  double* Qk = Qk_all + (size_t)mi * nbmax * kmax;
  const size_t tot = (size_t)nbmax * kmax;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int r = int(e % nbmax), q = int(e / nbmax);
    Qk[e] = (r < nb && q < k) ? Q[(size_t)(lo + W.qcol[lo + q]) * W.n + (lo + r)] : 0.0;
  }
}

// The batched product's columns and the deflated ones to their places in Qn.
__global__ void dc_scatter_kernel(DcWork W, int depth, int nbmax, int kmax, const double* __restrict__ Q,
                                  const double* __restrict__ Qm_all, double* __restrict__ Qn) {
  const int mi = blockIdx.y;
  const Span s = node_at(W.n, depth, mi);
  const int lo = s.lo, nb = s.hi - s.lo, k = W.counts[C_STRIDE * mi + C_K];
  const double* Qm = Qm_all + (size_t)mi * nbmax * kmax;
  const size_t tot = (size_t)nb * nb;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot; e += (size_t)gridDim.x * blockDim.x) {
    const int r = int(e % nb), t = int(e / nb);
    const double v = t < k ? Qm[r + (size_t)t * nbmax] : Q[(size_t)(lo + W.dcol[lo + t - k]) * W.n + (lo + r)];
    Qn[(size_t)(lo + W.outp[lo + t]) * W.n + (lo + r)] = v;
  }
}

// ---- the whole tree in one cluster -------------------------------------------------
__global__ void __launch_bounds__(kNT) dc_cluster_kernel(DcWork W, int levels, double* Q0, double* Q1) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) double dc_smem[];
  const int C = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  const int lane = threadIdx.x & 31, warp = rank * kNW + (threadIdx.x >> 5), nwarp = C * kNW;
  const int thread = rank * kNT + threadIdx.x, nthread = C * kNT;
  for (size_t e = thread; e < (size_t)W.n * W.n; e += nthread) Q0[e] = Q1[e] = 0.0;
  cluster.sync();
  for (int b = rank; b < (1 << levels); b += C) {
    const Span up = node_at(W.n, max(levels - 1, 0), b >> 1);
    Span s = node_at(W.n, levels, b);
    if (levels > 0 && up.hi - up.lo <= W.leaf) {
      if (b & 1) continue;
      s = up;
    }
    solve_leaf(W, s.lo, s.hi, Q0, Q1);
  }
  cluster.sync();
  double *Q = Q0, *Qn = Q1;
  for (int depth = levels - 1; depth >= 0; --depth) {
    const int nm = 1 << depth, nbmax = (W.n + nm - 1) >> depth;
    auto merges = [&](int mi) {
      const Span s = node_at(W.n, depth, mi);
      return s.hi - s.lo > W.leaf;
    };
    for (int mi = rank; mi < nm; mi += C) {
      const Span s = node_at(W.n, depth, mi);
      if (s.hi - s.lo > W.leaf)
        prep_merge(W, Q, s.lo, s.hi, mi, dc_smem);
      else if (threadIdx.x < C_STRIDE)
        W.counts[C_STRIDE * mi + threadIdx.x] = 0;
    }
    cluster.sync();
    const int lanes = secular_lanes(nm * nbmax, 4 * C);
    for (int g = rank + C * (threadIdx.x >> 5); g * (32 / lanes) < nm * nbmax; g += nwarp)
      secular_item(W, depth, nbmax, lanes, g, lane);
    cluster.sync();
    for (int mi = C - 1 - rank; mi < nm; mi += C) {
      const Span s = node_at(W.n, depth, mi);
      if (s.hi - s.lo > W.leaf) order_merge(W, s.lo, s.hi, mi, dc_smem);
    }
    for (int g = thread; g < nm * nbmax; g += nthread) {
      const int mi = g / nbmax, r = g % nbmax;
      const Span s = node_at(W.n, depth, mi);
      if (s.hi - s.lo > W.leaf && r < s.hi - s.lo && W.counts[C_STRIDE * mi + C_ROT] > 0)
        rotate_row(W, Q, s.lo, W.counts[C_STRIDE * mi + C_ROT], r);
    }
    for (int g = warp; g < nm * nbmax; g += nwarp) {
      const int mi = g / nbmax, j = g % nbmax;
      if (merges(mi) && j < W.counts[C_STRIDE * mi + C_K])
        gu_eisenstat(W, node_at(W.n, depth, mi).lo, W.counts[C_STRIDE * mi + C_K], j, W.rho[mi], lane,
                     W.Delta + (size_t)mi * nbmax * nbmax);
    }
    cluster.sync();
    for (int g = warp; g < nm * nbmax; g += nwarp) {
      const int mi = g / nbmax, i = g % nbmax;
      if (merges(mi) && i < W.counts[C_STRIDE * mi + C_K]) {
        const size_t o = (size_t)mi * nbmax * nbmax;
        secular_vector(W, node_at(W.n, depth, mi).lo, W.counts[C_STRIDE * mi + C_K], i, lane, W.Delta + o, W.St + o,
                       nbmax, 0);
      }
    }
    cluster.sync();
    const int per = merge_tiles(nbmax);
    for (int t = rank; t < nm * per; t += C) {
      const int mi = t / per;
      const Span s = node_at(W.n, depth, mi);
      if (s.hi - s.lo > W.leaf && t % per < merge_tiles(s.hi - s.lo))
        merge_tile(W, Q, Qn, s.lo, s.hi, mi, t % per, W.St + (size_t)mi * nbmax * nbmax, nbmax);
    }
    cluster.sync();
    double* x = Q;
    Q = Qn;
    Qn = x;
  }
}

// Orders that one cluster takes: measured, 16 CTAs win while their SMs hold the tree's
// levels (n = 96: 225 us against 272 in launches per step, 128: 274 against 301) and lose
// where another level and four times the merge work meet them (136: 458 against 360, 256:
// 759 against 436).
constexpr int kFusedMax = 128;

}  // namespace

// Leaf order: leaves are latency bound, so one solve is fastest with small leaves and more
// (batched) merge levels.  The context's override (4..32) trades that for fewer levels.
static int dc_leaf_size(const nsg_ctx* c) { return c->tune_dc_leaf > 0 ? c->tune_dc_leaf : 8; }

static int prep_smem(int nb) { return nb <= kSmemMerge ? nb * kPrepBytes : 0; }

static cudaLaunchConfig_t dc_cluster_config(nsg_ctx* c, int C, int smem, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(kNT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = C;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// CTAs of the cluster for order n: 4, 8 or 16 by the work there is, and no more than the
// device places together (a partition of it may hold fewer SMs side by side) or the context's
// override says; 0, a launch per step, where not even 4 are.
static int dc_cluster_size(nsg_ctx* c, int n) {
  if (c->dc_cluster == 0) {
    const auto fn = (const void*)dc_cluster_kernel;
    ensure_smem_limit(fn, prep_smem(kFusedMax));
    c->dc_cluster = 1;
    for (int C = 16; C >= 4 && c->dc_cluster == 1; C /= 2) {
      cudaLaunchAttribute attr[1];
      const cudaLaunchConfig_t cfg = dc_cluster_config(c, C, prep_smem(kFusedMax), attr);
      int fit = 0;
      const bool ok = (C <= 8 || cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                      cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) == cudaSuccess;
      if (ok && fit > 0) c->dc_cluster = C;
      if (!ok) cudaGetLastError();
    }
  }
  int C = n <= 32 ? 4 : n <= 64 ? 8 : 16;
  C = std::min(C, c->dc_cluster);
  if (c->tune_dc_cluster > 0) C = std::min(C, c->tune_dc_cluster);
  return C >= 4 ? C : 0;
}

double* tridiag_dc(nsg_ctx* c, int n, const double* d, const double* e, double* Q0, double* Q1, double* w, int* err) {
  DcWork W;
  W.n = n;
  W.leaf = dc_leaf_size(c);
  W.d = d;
  W.e = e;
  W.w = w;
  W.err = err;
  int levels = 0;
  while (((n + (1 << levels) - 1) >> levels) > W.leaf) ++levels;
  const int maxm = levels > 0 ? 1 << (levels - 1) : 1;
  // Delta and St: nm nbmax^2 entries at depth L, most at the top: nm nbmax <= n + nm
  size_t sq = 0;
  for (int L = 0; L < levels; ++L) {
    const size_t nm = size_t(1) << L, nb = (size_t(n) + nm - 1) >> L;
    sq = std::max(sq, nm * nb * nb);
  }
  const size_t N = (size_t(n) + 1) & ~size_t(1), MC = size_t(C_STRIDE) * maxm;
  const size_t doubles = 13 * N + 2 * sq + maxm + 2, ints = 9 * N + MC + 2;
  ScopedBuf buf(c, sizeof(double) * doubles + sizeof(int) * ints);
  double* p = (double*)buf.p;
  auto take = [&](size_t m) {
    double* q = p;
    p += m;
    return q;
  };
  W.Ds = take(N);
  W.zs = take(N);
  W.Dk = take(N);
  W.zk = take(N);
  W.wk = take(N);
  W.lam = take(N);
  W.zh = take(N);
  W.rot_cs = take(2 * N);
  W.gscr = take(4 * N);
  W.Delta = take(sq);
  W.St = take(sq);
  W.rho = take(maxm + 2);
  int* ip = (int*)p;
  auto takei = [&](size_t m) {
    int* q = ip;
    ip += m;
    return q;
  };
  W.perm = takei(N);
  W.kind = takei(N);
  W.qcol = takei(N);
  W.l1 = takei(N);
  W.l2 = takei(N);
  W.outp = takei(N);
  W.dcol = takei(N);
  W.low = takei(2);
  W.rot_pq = takei(2 * N);
  W.counts = takei(MC);
  if (const int C = n <= kFusedMax && levels > 0 ? dc_cluster_size(c, n) : 0) {
    ProfScope ps(c, NSG_PROF_DC, 0.0);
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = dc_cluster_config(c, C, prep_smem(n), attr);
    NSG_CUDA(cudaLaunchKernelEx(&cfg, dc_cluster_kernel, W, levels, Q0, Q1));
    count_launch(c);
    check_launch("dc cluster");
    return levels & 1 ? Q1 : Q0;
  }
  NSG_CUDA(cudaMemsetAsync(Q0, 0, sizeof(double) * n * n, c->stream));
  if (levels > 0) NSG_CUDA(cudaMemsetAsync(Q1, 0, sizeof(double) * n * n, c->stream));
  {
    ProfScope ps(c, NSG_PROF_DC, 0.0);
    dc_leaf_kernel<<<1 << levels, kNT, 0, c->stream>>>(W, levels, Q0, Q1);
  }
  count_launch(c);
  check_launch("dc leaves");
  double *Q = Q0, *Qn = Q1;
  for (int L = levels - 1; L >= 0; --L) {
    const int nm = 1 << L, nbmax = (n + nm - 1) >> L, shm = prep_smem(nbmax);
    // the merge product on the tensor cores in the split precision (the batched product
    // needs the largest kept count on the host); below 256 rows the FP64 tiles, which use
    // the halves' block structure, are faster than slicing the operands
    const bool tc = nbmax > 256 && (c->precision == NSG_PREC_OZAKI || c->precision == NSG_PREC_OZAKI8);
    const int gw = int((int64_t(nm) * nbmax * 32 + kNT - 1) / kNT);
    const int* cnt = nullptr;
    ensure_smem_limit((const void*)dc_prep_kernel, shm);
    const int oshm = nbmax <= kSmemMerge ? nbmax * 16 : 0;  // the orderings' part
    ensure_smem_limit((const void*)dc_weights_kernel, oshm);
    {
      ProfScope ps(c, NSG_PROF_DC, 0.0);
      dc_prep_kernel<<<nm, kNT, shm, c->stream>>>(W, L, Q);
      if (tc) {
        int* to = (int*)host_scalars(c, MC / 2 + 1);
        cnt = to;
        NSG_CUDA(cudaMemcpyAsync(to, W.counts, sizeof(int) * C_STRIDE * nm, cudaMemcpyDeviceToHost, c->stream));
        NSG_CUDA(cudaEventRecord(read_event(c), c->stream));
      }
      const int lanes = secular_lanes(nm * nbmax, 4 * c->num_sms);
      dc_secular_kernel<<<int((int64_t(nm) * nbmax * lanes + kNT - 1) / kNT), kNT, 0, c->stream>>>(W, L, nbmax, lanes);
      dc_weights_kernel<<<nm + nm * ((nbmax + kNT - 1) / kNT) + gw, kNT, oshm, c->stream>>>(W, L, nbmax, Q);
      dc_vectors_kernel<<<gw, kNT, 0, c->stream>>>(W, L, nbmax, tc);
      if (!tc) dc_merge_kernel<<<dim3(merge_tiles(nbmax), nm), kNT, 0, c->stream>>>(W, L, nbmax, Q, Qn);
    }
    count_launch(c, tc ? 4 : 5);
    check_launch("dc merge");
    if (tc) {
      // waits for the preparation's copy, not for the kernels launched since
      NSG_CUDA(cudaEventSynchronize(read_event(c)));
      int kmax = 0;
      for (int mi = 0; mi < nm; ++mi) kmax = std::max(kmax, cnt[C_STRIDE * mi + C_K]);
      ScopedBuf Qk(c, sizeof(double) * (size_t)nm * nbmax * std::max(kmax, 1)),
          Qm(c, sizeof(double) * (size_t)nm * nbmax * std::max(kmax, 1));
      const int per = std::max(1, c->num_sms * 8 / nm);
      if (kmax > 0) {
        {
          ProfScope ps(c, NSG_PROF_DC, 0.0);
          dc_gather_kernel<<<dim3(per, nm), 256, 0, c->stream>>>(W, L, nbmax, kmax, Q, (double*)Qk.p);
        }
        count_launch(c);
        GemmArgs g;
        g.dtype = NSG_F64;
        g.M = nbmax;
        g.N = kmax;
        g.K = kmax;
        g.A = Qk.p;
        g.lda = nbmax;
        g.opA = OP_N;
        g.strideA = (int64_t)nbmax * kmax;
        g.B = W.St;
        g.ldb = nbmax;
        g.opB = OP_N;
        g.strideB = (int64_t)nbmax * nbmax;
        g.C = Qm.p;
        g.ldc = nbmax;
        g.strideC = (int64_t)nbmax * kmax;
        g.batch = nm;
        gemm_accurate(c, g);
      }
      {
        ProfScope ps(c, NSG_PROF_DC, 0.0);
        dc_scatter_kernel<<<dim3(per, nm), 256, 0, c->stream>>>(W, L, nbmax, std::max(kmax, 1), Q, (const double*)Qm.p, Qn);
      }
      count_launch(c);
      check_launch("dc scatter");
    }
    std::swap(Q, Qn);
  }
  return Q;
}

}  // namespace nsg
