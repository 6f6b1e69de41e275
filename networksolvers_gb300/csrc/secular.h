// The scalar part of a secular root's iteration (dc.cu), and the word arithmetic it is written
// in: compiled for the device, and for the host, where it is tested by itself.
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define NSG_HD __host__ __device__ __forceinline__
#else
#define NSG_HD inline
#endif

namespace nsg {

constexpr double kEps = 2.220446049250313e-16;

NSG_HD long long bits_of(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  std::memcpy(&b, &x, sizeof b);
  return b;
#endif
}
NSG_HD double double_of(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
#endif
}
NSG_HD int high_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  return int(bits_of(x) >> 32);
#endif
}
NSG_HD double from_words(int hi, int lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, lo);
#else
  return double_of((long long)((unsigned long long)(unsigned)hi << 32 | (unsigned)lo));
#endif
}
NSG_HD double with_high_word(int hi, double x) {  // x with another high word
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, __double2loint(x));
#else
  return from_words(hi, int(bits_of(x)));
#endif
}

// Order-preserving integer key of a double (x < y exactly when key(x) < key(y); -0 and +0
// equal), so the merges compare with integer instructions rather than the FP64 pipe,
// and the exact negation -x by its sign bit.
NSG_HD long long order_key(double x) {
  const long long b = bits_of(x);
  if ((b & 0x7fffffffffffffffLL) == 0) return 0;
  return b < 0 ? (b ^ 0x7fffffffffffffffLL) : b;
}
NSG_HD double neg_exact(double x) { return double_of(bits_of(x) ^ (long long)(1ULL << 63)); }

// x 2^-e as a float (0 below its range), and x 2^e of a float as a double
NSG_HD float scaled_float(double x, int e) {
  const int hi = high_word(x), ex = ((hi >> 20) & 0x7ff) - e;
  return ex <= 0 || ex >= 0x7ff ? 0.f : (float)with_high_word(hi - (e << 20), x);
}
NSG_HD double scaled_double(float x, int e) {
  const double d = (double)x;
  const int ex = ((high_word(d) >> 20) & 0x7ff) + e;
  return x == 0.f || ex <= 0 || ex >= 0x7ff ? 0.0 : with_high_word(high_word(d) + (e << 20), d);
}

// Root i of 1 + sum_j w_j / (D_j - lambda), w_j = rho z_j^2, lies in (D_i, D_{i+1}) (the last
// one in (D_{k-1}, D_{k-1} + rho)); it is represented as origin + tau with the origin at the
// nearer pole, so D_j - lambda = (D_j - origin) - tau is exact enough for the recomputed
// weights.  The first evaluation, at the interval's middle, chooses the origin and also feeds
// the first step.  Steps: the two-pole rational model with the origin's weight kept (R.-C. Li,
// LAPACK Working Note 89, 1994), solved in FP32, and bisection of the bracket (of its exponent
// where it spans binades) when that leaves it or |f| grew: up to 5 evaluations for 94 % of random,
// graded and clustered roots, up to 8 for 98.6 %.  On two close poles under a distant one the
// model can creep without |f| growing (six roots in ten million of random clustered problems had
// not arrived after 100 steps, some with |f| of order one): from step kSecularBisect on every
// step bisects, and over 300 million such roots none takes more than 84.  (The start is written
// out in dc.cu: as a member it cost the divide and conquer of order 128 1.5 %.)
constexpr int kSecularBisect = 30, kSecularSteps = 128;
struct SecularRoot {
  double dorg, tau, blo, bhi;  // origin, and the root and its bracket relative to it
  double q1, q2;               // the model's poles relative to the origin: i and i + 1, or the two last
  double worg;                 // the origin's weight: its pole enters with it, the other pole with the
                               // rest of the slope
  float ftol, fprev;           // 4 eps (k + 1); |f| of the step before (infinite at first)
  int jorg;                    // the origin's pole
  bool inner, left, single;    // not the last root; the origin is pole i; k = 1

  // The step after evaluation `it`: f, its slope dr (without the origin pole's part but for the
  // first), fa the sum of its terms' magnitudes.  Returns whether tau is the root.
  template <typename Recip, typename Divide>
  NSG_HD bool step(int it, double f, double dr, float fa, Recip recip, Divide divide) {
    if (high_word(f) >= 0)
      bhi = tau;
    else
      blo = tau;
    const float ff = (float)f;
    double tn = tau;
    bool done = fabsf(ff) <= fmaf(ftol, fa, ftol);
    if (it >= 5 && !done) done = bhi - blo <= 2.0 * kEps * fmax(fabs(blo), fabs(bhi)) || bhi - blo < 1e-300;
    if (!done) {
      // |f| grew (or, for the last root under many poles, has halved slowly three times)
      const bool slow = it >= kSecularBisect ||
                        (inner ? it >= 2 && fabsf(ff) > fprev : it >= 3 && fabsf(ff) > 0.5f * fprev);
      fprev = fabsf(ff);
      // the increment in FP32, lengths scaled by the farther pole's distance: it needs a
      // few digits only, the next evaluation is in FP64 again
      const double p1 = q1 - tau, p2 = q2 - tau;
      const int e1 = (high_word(p1) >> 20) & 0x7ff, e2 = (high_word(p2) >> 20) & 0x7ff, e = (e1 > e2 ? e1 : e2) - 1023;
      const float t = scaled_float(tau, e), u1 = scaled_float(p1, e), u2 = scaled_float(p2, e);
      const float r = divide(1.f, t), w1 = scaled_float(worg, e) * r * r;
      const float s1 = scaled_float(dr, -e) - (it == 0 ? w1 : 0.f);  // the other poles' slope
      // x: the increment, the root of c x^2 - a x + b = 0; y: the new distance from the
      // origin directly, the root of c y^2 - h y + w q = 0 (for steps that take tau nearly
      // to the origin, where the increment would cancel)
      float x, y;
      if (inner || !single) {
        const float uo = inner && left ? u2 : u1;  // the other pole
        const float pr = u1 * u2, a = fmaf(-pr, s1 + w1, (u1 + u2) * ff), b = pr * ff;
        float c = fmaf(-uo, s1, fmaf(t, w1, ff));
        if (!inner) c = fabsf(c);
        const float v = a + copysignf(sqrtf(fmaxf(fmaf(a, a, -4.f * b * c), 0.f)), a);
        x = (a < 0.f) == inner ? 0.5f * v / c : 2.f * b / v;
        const float q = uo + t, w = w1 * t * t, h = fmaf(c, q, fmaf(s1 * uo, uo, w));
        const float z = h + copysignf(sqrtf(fmaxf(fmaf(h, h, -4.f * c * w * q), 0.f)), h);
        y = (h >= 0.f) == inner ? 2.f * w * q / z : 0.5f * z / c;
      } else {  // one pole
        x = -t * ff / fmaf(t, w1, ff);
        y = t + x;
      }
      // (not a step downhill, not a number, or lost to FP32's range: Newton's step)
      if (x * ff < 0.f && fabsf(x) < 1e30f)
        tn = fabsf(x) > 0.5f * fabsf(t) && y * t > 0.f ? scaled_double(y, e) : tau + scaled_double(x, e);
      else
        tn = tau - f * recip(dr + (it == 0 ? 0.0 : scaled_double(w1, -e)));
      const long long kt = order_key(tn);
      if (!(tn == tn) || kt <= order_key(blo) || kt >= order_key(bhi) || slow) {
        // out of the bracket, or slow: bisect, in the exponent where the bracket spans
        // several binades
        const long long ml = bits_of(blo) & 0x7fffffffffffffffLL, mh = bits_of(bhi) & 0x7fffffffffffffffLL;
        const int em = int((ml < mh ? ml : mh) >> 52), eM = int((ml < mh ? mh : ml) >> 52);
        tn = 0.5 * (blo + bhi);
        if (em == 0 && it >= 2 && eM > 40)
          tn = from_words((eM - 10) << 20, 0);
        else if (em > 0 && eM - em > 6)
          tn = from_words(((em + eM) / 2) << 20, 0);
        if (high_word(blo) < 0 && tn > 0.0) tn = neg_exact(tn);
      }
      done = tn == tau;
    }
    tau = tn;
    return done;
  }
};

}  // namespace nsg
