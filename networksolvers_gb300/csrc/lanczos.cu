// The vector work of a Lanczos step in one cooperative launch (krylov.cu holds the
// recurrence): w -= beta v_{j-1}, two classical Gram-Schmidt passes against v_0 .. v_j, the
// sum of squares of what is left and the next basis vector, with every scalar on the device.
// Each of the three sums is reduced within the CTA, published in 16-byte messages that carry
// a tag beside the value, and gathered by every CTA (in CTA order: the sums are the same
// everywhere and from run to run), so that no launch ends for a scalar.  A thread keeps its
// elements through all passes, and re-reads only what it wrote itself.
//
// Bound: FP64 operations for long vectors (4 nv + 2 an element; a warp-wide one holds its SM
// sub-partition for 64 cycles), about 3000 cycles per sum for short ones.  As separate launches
// (a dot product's two, an update, a dot product's two, ..) a step takes 9 or 10: the region
// step at bond dimension 64 (16384 elements, three steps) 1194 us with them and 1082 with this,
// the eigensolve at bond dimension 1024 (4.2 million) 6.76 and 6.54 ms, a two-site TDVP step at
// 128 (complex) 7.65 and 6.83.
#include "nsg_internal.h"
#include "tagged.h"

#include <algorithm>

namespace nsg {

namespace {

constexpr int kT = 256, kW = kT / 32;
constexpr int kMaxVec = 16;              // vectors of a step; more take separate launches
constexpr int kVals = 2 * kMaxVec;       // doubles of a sum, at most
constexpr int kPollDelay = 400;          // cycles from publishing to the first poll (polls slow the stores)

struct Step {
  const void* v[kMaxVec];
  int nv;
  int64_t n;
  void* w;             // updated in place (nv = 0: only read)
  void* next;          // w / sqrt(sum of squares), or null
  const double* prev;  // ss of the step before (w -= sqrt(.) v[nv - 2] first), or null
  double *co1, *co2, *ss;  // coefficients; the sum of squares and its root
  ulonglong2* msg;     // 3 sums x CTAs x kVals
  unsigned long long tag;
  int polls;           // of a wait before it gives up; below 0 it does so at once
  int* gave_up;
};

__device__ __forceinline__ double fnma(double a, double v, double w) { return fma(-a, v, w); }
__device__ __forceinline__ double2 fnma(double2 a, double2 v, double2 w) {
  return make_double2(fma(a.y, v.y, fma(-a.x, v.x, w.x)), fma(-a.y, v.x, fma(-a.x, v.y, w.y)));
}
// s + conj(v) w
__device__ __forceinline__ double dot(double s, double v, double w) { return fma(v, w, s); }
__device__ __forceinline__ double2 dot(double2 s, double2 v, double2 w) {
  return make_double2(fma(v.x, w.x, fma(v.y, w.y, s.x)), fma(v.x, w.y, fma(-v.y, w.x, s.y)));
}
__device__ __forceinline__ double sumsq(double s, double w) { return fma(w, w, s); }
__device__ __forceinline__ double sumsq(double s, double2 w) { return fma(w.x, w.x, fma(w.y, w.y, s)); }
__device__ __forceinline__ double times(double a, double w) { return a * w; }
__device__ __forceinline__ double2 times(double a, double2 w) { return make_double2(a * w.x, a * w.y); }
__device__ __forceinline__ double real_coef(double, double a) { return a; }
__device__ __forceinline__ double2 real_coef(double2, double a) { return make_double2(a, 0.0); }

// The sums over a warp of NV doubles per lane, to part[0 .. NV): the first levels of the
// butterfly halve the values a lane holds
template <int NV>
__device__ __forceinline__ void warp_sums(const double* in, int lane, double* part) {
  constexpr int NP = NV > 4 ? 8 : NV > 2 ? 4 : NV;
  double a[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) a[i] = i < NV ? in[i] : 0.0;
  int o = 16;
#pragma unroll
  for (int h = NP / 2; h >= 1; h /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double send = up ? a[i] : a[i + h], keep = up ? a[i + h] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o > 0; o /= 2) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
  constexpr int kLow = 32 / NP;
  if (lane % kLow == 0 && lane / kLow < NV) part[lane / kLow] = a[0];
}

// The sums of part[warp][0 .. nvals) over the warps and the CTAs, to res[0 .. nvals) (shared).
// area: which of the launch's sums.
__device__ void all_sums(const Step& s, int area, int nvals, const double (*part)[kVals], double* res) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
  __syncthreads();
  ulonglong2* msg = s.msg + (size_t)area * G * kVals;
  if (tid < nvals) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kW; ++w) t += part[w][tid];
    if (G == 1)
      res[tid] = t;
    else
      put_tagged(msg + (size_t)tid * G + blockIdx.x, t, s.tag + area);
  }
  if (G > 1) {
    for (const long long t0 = clock64(); clock64() - t0 < kPollDelay;) {
    }
    for (int q = warp; q < nvals; q += kW) {
      double t = 0.0;
      for (int b = lane; b < G; b += 32) {
        double x = 0.0;
        int polls = s.polls;
        bool there = false;
        while (polls-- > 0 && !there) there = get_tagged(msg + (size_t)q * G + b, s.tag + area, x);
        if (!there) {
          atomicExch(s.gave_up, 1);
          x = __longlong_as_double(0x7ff8000000000000ll);
        }
        t += x;
      }
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) res[q] = t;
    }
  }
  __syncthreads();
}

// NV: the vectors, all held in registers while an element is updated and entered into the
// next sums; 0: any number up to kMaxVec, in groups of four.
template <typename T, int NV>
__global__ void __launch_bounds__(kT, 2) lanczos_step_kernel(const __grid_constant__ Step s) {
  constexpr bool cplx = sizeof(T) == 16;
  constexpr int E = cplx ? 2 : 1, U = cplx ? 2 : 4;
  __shared__ double part[kW][kVals], res[kVals];
  __shared__ T coef[kMaxVec];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t stride = (int64_t)gridDim.x * kT, first = blockIdx.x * (int64_t)kT + tid;
  T* w = (T*)s.w;
  const int nv = NV ? NV : s.nv;
  // f(element index, w's value) -> w's new value, over the thread's elements, U at a time
  auto sweep = [&](bool store, auto&& load, auto&& f) {
    for (int64_t i0 = first; i0 < s.n; i0 += U * stride) {
      T x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = i0 + u * stride < s.n ? w[i0 + u * stride] : T{};
      load(i0);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * stride < s.n) {
          const T y = f(u, i0 + u * stride, x[u]);
          if (store) w[i0 + u * stride] = y;
        }
    }
  };
  if constexpr (NV > 0) {
    T v[NV][U], acc[NV];
    auto load = [&](int64_t i0) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int u = 0; u < U; ++u)
          v[k][u] = i0 + u * stride < s.n ? ((const T*)s.v[k])[i0 + u * stride] : T{};
    };
    auto reduce = [&](int area, double* out) {
      warp_sums<E * NV>((const double*)acc, lane, part[warp]);
      all_sums(s, area, E * NV, part, res);
      if (tid < NV) {
        if constexpr (cplx)
          coef[tid] = make_double2(res[2 * tid], res[2 * tid + 1]);
        else
          coef[tid] = res[tid];
        if (blockIdx.x == 0) {
          out[2 * tid] = res[E * tid];
          out[2 * tid + 1] = cplx ? res[E * tid + E - 1] : 0.0;
        }
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] = T{};
    };
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = T{};
    const bool sub = NV > 1 && s.prev;
    const T b = real_coef(T{}, sub ? s.prev[1] : 0.0);
    sweep(sub, load, [&](int u, int64_t, T x) {
      if (sub) x = fnma(b, v[NV > 1 ? NV - 2 : 0][u], x);
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] = dot(acc[k], v[k][u], x);
      return x;
    });
    reduce(0, s.co1);
    T c[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) c[k] = coef[k];
    sweep(true, load, [&](int u, int64_t, T x) {
#pragma unroll
      for (int k = 0; k < NV; ++k) x = fnma(c[k], v[k][u], x);
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] = dot(acc[k], v[k][u], x);
      return x;
    });
    reduce(1, s.co2);
#pragma unroll
    for (int k = 0; k < NV; ++k) c[k] = coef[k];
    double ss = 0.0;
    sweep(true, load, [&](int u, int64_t, T x) {
#pragma unroll
      for (int k = 0; k < NV; ++k) x = fnma(c[k], v[k][u], x);
      ss = sumsq(ss, x);
      return x;
    });
    warp_sums<1>(&ss, lane, part[warp]);
  } else {
    const auto none = [](int64_t) {};
    if (nv > 1 && s.prev) {
      const T b = real_coef(T{}, s.prev[1]);
      const T* v = (const T*)s.v[nv - 2];
      sweep(true, none, [&](int, int64_t i, T x) { return fnma(b, v[i], x); });
    }
    for (int pass = 0; pass < 2 && nv > 0; ++pass) {
      for (int g = 0; g < nv; g += 4) {
        T acc[4] = {};
        const T* v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (const T*)s.v[min(g + k, nv - 1)];
        sweep(false, none, [&](int, int64_t i, T x) {
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[k] = dot(acc[k], v[k][i], x);
          return x;
        });
        warp_sums<4 * E>((const double*)acc, lane, part[warp] + E * g);
      }
      all_sums(s, pass, E * nv, part, res);
      if (tid < nv) {
        if constexpr (cplx)
          coef[tid] = make_double2(res[2 * tid], res[2 * tid + 1]);
        else
          coef[tid] = res[tid];
        if (blockIdx.x == 0) {
          double* out = pass ? s.co2 : s.co1;
          out[2 * tid] = res[E * tid];
          out[2 * tid + 1] = cplx ? res[E * tid + E - 1] : 0.0;
        }
      }
      __syncthreads();
      sweep(true, none, [&](int, int64_t i, T x) {
        for (int k = 0; k < nv; ++k) x = fnma(coef[k], ((const T*)s.v[k])[i], x);
        return x;
      });
    }
    double ss = 0.0;
    sweep(false, none, [&](int, int64_t, T x) {
      ss = sumsq(ss, x);
      return x;
    });
    warp_sums<1>(&ss, lane, part[warp]);
  }
  all_sums(s, 2, 1, part, res);
  if (warp == 0) {  // (by one warp: the root and the quotient are ten FP64 operations each)
    const double root = sqrt(res[0]);
    if (lane == 0) {
      res[1] = 1.0 / root;
      if (blockIdx.x == 0) {
        s.ss[0] = res[0];
        s.ss[1] = root;
      }
    }
  }
  __syncthreads();
  // (normalised in place: a CTA whose wait gave up leaves its part as it is)
  if (s.next && (s.next != s.w || isfinite(res[0]))) {
    const double a = res[1];
    T* next = (T*)s.next;
    sweep(false, [](int64_t) {}, [&](int, int64_t i, T x) {
      next[i] = times(a, x);
      return x;
    });
  }
}

template <typename T>
const void* step_kernel(int nv) {
  switch (nv) {
    case 1: return (const void*)lanczos_step_kernel<T, 1>;
    case 2: return (const void*)lanczos_step_kernel<T, 2>;
    case 3: return (const void*)lanczos_step_kernel<T, 3>;
    case 4: return (const void*)lanczos_step_kernel<T, 4>;
    default: return (const void*)lanczos_step_kernel<T, 0>;
  }
}

}  // namespace

LanczosVectors::LanczosVectors(nsg_ctx* ctx, int dt, int64_t len, int* gave_up_flag)
    : c(ctx), dtype(dt), n(len), gave_up(gave_up_flag) {
  // every CTA gathers every CTA's sums, so no more CTAs than pay: a CTA has at least 512
  // elements (2048 instead: TDVP step at bond dimension 128 7 % slower), one CTA per SM, and two
  // from 2^21 elements on, where the loads in flight count (eigensolve at bond dimension 1024,
  // 4.2 million: 6.56 ms against 6.65; two at 240000 elements: 5.315 against 5.299)
  const int64_t sms = std::max(c->num_sms, 1);
  grid = int(std::min<int64_t>(n >= (int64_t(1) << 21) ? 2 * sms : sms, std::max<int64_t>(1, (n + 511) / 512)));
  if (grid > 1) {
    bytes = sizeof(ulonglong2) * 3 * size_t(grid) * kVals;
    msg = dalloc(c, bytes);
    NSG_CUDA(cudaMemsetAsync(msg, 0, bytes, c->stream));
  }
}
LanczosVectors::~LanczosVectors() {
  try {
    if (msg) dfree(c, msg, bytes);
  } catch (...) {
  }
}

bool LanczosVectors::step(int nv, const void* const* v, void* w, const double* prev, double* co1, double* co2, double* ss,
                          void* next) {
  if (nv > kMaxVec) return false;
  Step s{};
  for (int j = 0; j < nv; ++j) s.v[j] = v[j];
  s.nv = nv;
  s.n = n;
  s.w = w;
  s.next = next;
  s.prev = prev;
  s.co1 = co1;
  s.co2 = co2;
  s.ss = ss;
  s.msg = (ulonglong2*)msg;
  s.tag = tag;
  tag += 4;
  const int polls = c->tune_lanczos_polls;
  s.polls = polls == -2 ? (next == w ? -1 : 1 << 22) : polls != 0 ? polls : 1 << 22;
  s.gave_up = gave_up;
  const void* fn = dtype == NSG_C128 ? step_kernel<double2>(nv) : step_kernel<double>(nv);
  void* args[] = {&s};
  NSG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kT), args, 0, c->stream));
  count_launch(c);
  check_launch("lanczos step");
  return true;
}

}  // namespace nsg
