"""The secular roots' iteration (csrc/secular.h) compiled for the host, its sums in plain double
precision as the device forms them: every root is found within the loop's bound, to the stopping
rule's residual (4 eps (k + 1) times the sum of the terms' magnitudes; twice that, for the sums'
own rounding) or, where that is out of reach, to 4 eps of itself."""
import subprocess

import pytest

from networksolvers_gb300 import build as nb

MAIN = r"""
#include "secular.h"
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <iostream>
#include <vector>
using namespace nsg;
using Vec = std::vector<double>;
static long long failed = 0;
static int steps = 0;

static void check(const Vec& D, const Vec& w, double rho, int i) {
  const int k = int(D.size());
  const double gap = i < k - 1 ? D[i + 1] - D[i] : 0.0;
  SecularRoot r;
  r.dorg = D[i];
  double f, dr;
  float fa;
  auto eval = [&](double tau, int skip) {
    double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
    for (int j = 0; j < k; ++j) {
      const double q = 1.0 / ((D[j] - r.dorg) - tau), a = w[j] * q, b = j == skip ? 0.0 : a * q;
      (j <= i ? psi : phi) += a;
      (j <= i ? dpsi : dphi) += b;
    }
    f = 1.0 + (psi + phi);
    dr = dpsi + dphi;
    fa = fabsf((float)psi - (float)phi);
  };
  // the start as the device makes it
  r.inner = i < k - 1;
  r.single = k <= 1;
  r.blo = 0.0;
  r.bhi = r.inner ? gap : rho;
  r.tau = 0.5 * r.bhi;
  eval(r.tau, -1);
  r.left = true;
  if (r.inner && f >= 0) {
    r.bhi = r.tau;
  } else if (r.inner) {
    r.left = false;
    r.dorg = D[i + 1];
    r.tau = -r.tau;
    r.blo = r.tau;
    r.bhi = 0.0;
  }
  r.ftol = float(4.0 * kEps) * float(k + 1);
  r.fprev = INFINITY;
  r.q1 = r.inner ? (r.left ? 0.0 : -gap) : (r.single ? 0.0 : D[k - 2] - r.dorg);
  r.q2 = r.inner && r.left ? gap : 0.0;
  r.jorg = r.inner && !r.left ? i + 1 : i;
  r.worg = w[r.jorg];
  bool done = false;
  int it = 0;
  for (; it < kSecularSteps && !done; ++it) {
    if (it > 0) eval(r.tau, r.jorg);
    done = r.step(it, f, dr, fa, [](double d) { return 1.0 / d; }, [](float a, float b) { return a / b; });
  }
  steps = std::max(steps, it);
  long double mag = 1.0L;
  auto F = [&](long double t) {
    long double s = 1.0L;
    mag = 1.0L;
    for (int j = 0; j < k; ++j) {
      const long double a = w[j] / (((long double)D[j] - r.dorg) - t);
      s += a;
      mag += fabsl(a);
    }
    return s;
  };
  const long double res = fabsl(F(r.tau));
  const bool small = res <= 8.0L * kEps * (k + 1) * mag;
  const long double lo = F(r.tau - 4 * kEps * fabs(r.tau)), hi = F(r.tau + 4 * kEps * fabs(r.tau));
  if (!done || !(small || lo * hi <= 0)) {
    if (failed++ < 5) printf("k %d root %d rho %g: done %d residual %Lg\n", k, i, rho, done, res);
  }
}

static uint64_t state = 1;
static double uniform() {  // xorshift64*
  state ^= state >> 12;
  state ^= state << 25;
  state ^= state >> 27;
  return double((state * 2685821657736338717ull) >> 11) * 0x1p-53;
}

int main() {
  int n;
  std::cin >> n;
  while (n--) {
    int k, i;
    double rho;
    std::cin >> k;
    Vec D(k), w(k);
    for (double& x : D) std::cin >> x;
    for (double& x : w) std::cin >> x;
    std::cin >> rho >> i;
    check(D, w, rho, i);
  }
  // random, graded and clustered poles, weights of one size or graded, coupling far below to far
  // above the poles, deflated as the merges do
  for (int q = 0; q < 60000; ++q) {
    const int k = 1 + int(pow(40.0, uniform())), kind = q % 8;
    Vec p(k), z(k);
    const double span = 16 * uniform();
    double nz = 0.0;
    for (int j = 0; j < k; ++j) {
      const double u = uniform();
      p[j] = kind % 4 == 0   ? 2 * u - 1
             : kind % 4 == 1 ? pow(10.0, -span * u) * (uniform() < 0.5 ? 1 : -1)
             : kind % 4 == 2 ? floor(4 * uniform()) + pow(10.0, -15 * u)
                             : 1.0 + 1e-10 * u;
      z[j] = kind >= 4 ? pow(10.0, -15.5 * uniform()) : 2 * uniform() - 1;
      nz += z[j] * z[j];
    }
    std::sort(p.begin(), p.end());
    const double top = std::max(fabs(p[0]), fabs(p[k - 1])), rho = pow(10.0, 17 * uniform() - 14) * top;
    const double tol = 8 * kEps * std::max(top, rho);
    Vec D, w;
    for (int j = 0; j < k; ++j) {
      const double v = z[j] / sqrt(nz);
      if (rho * fabs(v) <= tol || (!D.empty() && p[j] - D.back() <= tol)) continue;
      D.push_back(p[j]);
      w.push_back(rho * v * v);
    }
    for (int i = 0; i < int(D.size()); ++i) check(D, w, rho, i);
  }
  printf("failed %lld, steps at most %d\n", failed, steps);
}
"""

# pairs of close poles under a distant one, on which the model's steps creep: poles, weights
# (rho z^2), rho, root
CREEPING = [
    ([1.0000000000006484, 1.000000000000689, 2.000000000000079],
     [9.4044922799626144e-11, 9.1880600388670141e-11, 5.1835953237481714e-11], 2.37761476425778e-10, 1),
    ([3.54697853612728e-13, 7.1898464993872117e-13, 1.0000000000000902, 1.0269800325627891],
     [5.504792254701895e-12, 4.7486778889497644e-12, 1.5808514056402069e-11, 3.6865600400081255e-12],
     2.974854424006185e-11, 1),
    ([6.7420312531746876e-14, 2.6317015085330811e-12, 2.0000000000000049, 2.0005973338713288],
     [1.6557734323633643e-09, 1.6512823224747427e-09, 8.4828164971682371e-10, 4.0722942483566808e-10],
     4.5625668293905991e-09, 1),
    ([7.4400789650723419e-07, 1.0003101103559966, 2.0000000000863993, 2.0000000001428737, 3.0000000479458926],
     [1.6913908086185743e-14, 4.7509171145823889e-12, 5.9223147387263108e-10, 4.7800315909773364e-10,
      6.4357546871961514e-10], 1.7185779327126484e-09, 3),
    ([5.3996172393836552e-13, 1.0000000000000431, 1.0000000000000644, 2.0000000000020997],
     [2.2864508123779826e-13, 1.4800229078383717e-13, 1.1302066675065618e-13, 5.283444463810108e-12],
     5.7731125025823998e-12, 2),
]


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    d = tmp_path_factory.mktemp("secular")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", f"-I{nb.CSRC}", str(d / "main.cpp"), "-o",
                    str(d / "main")], check=True)
    words = [len(CREEPING)]
    for D, w, rho, i in CREEPING:
        words += [len(D), *D, *w, rho, i]
    return subprocess.run([str(d / "main")], input=" ".join(map(repr, words)), capture_output=True, text=True,
                          check=True).stdout


def test_every_root_is_found(report):
    assert "failed 0," in report, report
