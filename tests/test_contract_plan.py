"""The contraction planner (csrc/contract_plan.h, host code) compiled by itself: the trees it
finds are flop-optimal, and it stays quick where almost every tree ties."""
import itertools
import math
import subprocess
from pathlib import Path

import pytest

from networksolvers_gb300 import build as nb
from networksolvers_gb300._native import PRECISIONS

MAIN = r"""
#include "contract_plan.h"
#include <chrono>
#include <cstdio>
#include <iostream>
int main() {
  int nets;
  std::cin >> nets;
  for (int q = 0; q < nets; ++q) {
    auto list = [] {
      int k;
      std::cin >> k;
      std::vector<int> v(k);
      for (int& x : v) std::cin >> x;
      return v;
    };
    int n, precision;
    std::cin >> n >> precision;
    std::vector<std::vector<int>> labs(n);
    for (auto& l : labs) l = list();
    const std::vector<int> out = list(), names = list(), sizes = list();
    std::unordered_map<int, int64_t> dims;
    for (size_t k = 0; k < names.size(); ++k) dims[names[k]] = sizes[k];
    double best = 1e30;
    nsg::Tree t;
    try {
      for (int rep = 0; rep < 2; ++rep) {
        const auto t0 = std::chrono::steady_clock::now();
        t = nsg::optimal_tree(labs, out, dims, precision);
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
      }
    } catch (const nsg::Error& e) {
      printf("error %d\n", e.code);
      continue;
    }
    int rank = 0;
    for (const auto& nd : t.nodes) rank = std::max(rank, nd.order.n);
    printf("%.17g %.17g %g %d %.17g\n", t.total_macs, t.moved, best, rank, t.fp64_macs);
  }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    cuda = Path(nb.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", f"-I{nb.CSRC}", f"-I{cuda}", str(d / "main.cpp"), "-o",
                    str(d / "main")], check=True)

    def run(nets, precision=PRECISIONS["fp64"]):
        words = [len(nets)]
        for labs, out, dims in nets:
            words += [len(labs), precision]
            for x in (*labs, out, list(dims), list(dims.values())):
                words += [len(x), *x]
        r = subprocess.run([str(d / "main")], input=" ".join(map(str, words)), capture_output=True, text=True,
                           check=True)
        return [[float(v) for v in line.split()] if line[0] != "e" else line for line in r.stdout.splitlines()]
    return run


def heff(a, b, w=5):
    """L W1 W2 R x of a two-site region with left bond a and right bond b."""
    dims = {0: a, 1: a, 2: w, 3: 2, 4: 2, 5: w, 6: 2, 7: 2, 8: w, 9: b, 10: b}
    return [[1, 2, 0], [10, 8, 9], [2, 4, 3, 5], [5, 7, 6, 8], [0, 3, 6, 9]], [1, 4, 7, 10], dims


def env(z, chi, w=5):
    """The environment update at a vertex of z bonds."""
    A, W, B = [0, *range(10, 10 + z)], [1, 0, *range(30, 30 + z)], [1, *range(50, 50 + z)]
    dims = {0: 2, 1: 2}
    for i in range(z):
        dims.update({10 + i: chi, 30 + i: w, 50 + i: chi})
    return [A, *([50 + i, 30 + i, 10 + i] for i in range(z - 1)), W, B], [49 + z, 29 + z, 9 + z], dims


def chain(n, d):
    return [[l for l in (i - 1, i) if 0 <= l < n - 1] for i in range(n)], [], {i: d for i in range(n - 1)}


def star(n, d):
    return [list(range(n - 1)), *([i] for i in range(n - 1))], [], {i: d for i in range(n - 1)}


def least_macs(net):
    """Fewest multiply-adds of any pairwise order, by the recurrence over subsets."""
    labs, out, dims = net
    full = frozenset(range(len(labs)))

    def is_open(S):
        inside, outside = {l for i in S for l in labs[i]}, {l for i in full - S for l in labs[i]} | set(out)
        return inside & outside

    cost = {frozenset([i]): 0 for i in full}
    for k in range(2, len(labs) + 1):
        for S in map(frozenset, itertools.combinations(sorted(full), k)):
            first = min(S)
            rest = sorted(S - {first})
            cost[S] = min(cost[P] + cost[S - P] + math.prod(dims[l] for l in is_open(P) | is_open(S - P))
                          for r in range(len(rest)) for P in (frozenset((first, *c)) for c in
                                                              itertools.combinations(rest, r)))
    return cost[full]


def test_orders_are_flop_optimal(plan):
    nets = [heff(64, 64), heff(60, 240), heff(7, 300, 14), env(2, 100), env(3, 32), env(4, 8), env(5, 6), chain(6, 3),
            star(7, 4), chain(7, 1)]
    for net, got in zip(nets, plan(nets)):
        assert got[0] == least_macs(net)


def test_a_chain_region_permutes_operator_tensors_only(plan):
    # (two of the W tensors, 100 elements each, and their launches)
    for got in plan([heff(64, 64), heff(60, 240), heff(475, 475)]):
        assert got[1] < 2 * (2e4 + 101)


def test_ties_do_not_blow_the_planning_up(plan):
    # 6 ms, where a search of every tie takes 0.4 to 60 s
    nets = [chain(12, 1), star(12, 1), star(12, 4), chain(10, 1), star(10, 1)]
    for net, got in zip(nets, plan(nets)):
        assert got[0] == len(net[0]) - 1 or 4 in net[2].values()
        assert got[2] < 0.15


def test_intermediates_fit_a_tensors_rank(plan):
    # trees of equal flops, some of them through an intermediate of more than 16 labels
    labs = [[9, 8, 5, 3, 1, 6, 0, 7, 2, 4],
            [0, 15, 16, 18, 12, 25, 17, 14, 1, 13, 10, 11],
            [21, 10, 2, 22, 3, 19, 20, 11, 26],
            [13, 19, 4, 27, 24, 23, 12, 20],
            [16, 5, 24, 7, 15, 6, 14, 23],
            [21, 8, 18, 22, 17, 9]]
    two = [2, 5, 6, 7, 8, 9, 10, 12, 17, 19]
    net = labs, [25, 26, 27], {l: 2 if l in two else 1 for t in labs for l in t}
    got, wide = plan([net, ([[*range(10)], [*range(10, 20)]], [*range(20)], dict.fromkeys(range(20), 1))])
    assert got[3] <= 16 and got[0] == least_macs(net)
    assert wide == "error 7"


def test_ties_keep_products_on_the_tensor_cores(plan):
    """H_eff applications in the split precision: in one of the mirrored orders all but the two
    operator tensors' products (5 x 2 x 5 x 2 of each of 2 a b entries) meet its least sizes."""
    shapes = [(60, 240), (63, 100), (60, 1000), (100, 63), (240, 60), (128, 128)]
    for (a, b), got in zip(shapes, plan([heff(a, b) for a, b in shapes], PRECISIONS["ozaki"])):
        assert got[4] == 2 * 100 * 2 * a * b, (a, b)
