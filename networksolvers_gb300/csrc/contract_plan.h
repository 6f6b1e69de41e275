// Planning of tensor-network contractions (contract.cu runs the plans): how two labelled
// operands become one (strided-batched) product, and in which pairwise order a network is
// contracted.  Host code without device calls.
#pragma once

#include "nsg_internal.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <unordered_map>
#include <vector>

namespace nsg {

// A short list of labels without an allocation (the planning below forms thousands).
struct Labs {
  int n = 0;
  int v[2 * NSG_MAX_RANK];
  Labs() {}
  Labs(const std::vector<int>& x) {
    NSG_CHECK(x.size() <= 2 * NSG_MAX_RANK, NSG_ERR_UNSUPPORTED, "contract: result rank above 16");
    for (int l : x) push_back(l);
  }
  void push_back(int l) {
    NSG_CHECK(n < 2 * NSG_MAX_RANK, NSG_ERR_UNSUPPORTED, "contract: result rank above 16");
    v[n++] = l;
  }
  void append(const Labs& o, int from, int to) {
    for (int k = from; k < to; ++k) push_back(o.v[k]);
  }
  const int* begin() const { return v; }
  const int* end() const { return v + n; }
  int at(int l) const {
    for (int k = 0; k < n; ++k)
      if (v[k] == l) return k;
    return -1;
  }
  bool operator==(const Labs& o) const { return n == o.n && std::equal(v, v + n, o.v); }
  bool operator!=(const Labs& o) const { return !(*this == o); }
  std::vector<int> list() const { return std::vector<int>(v, v + n); }
};

// Where the contracted labels sit inside an operand: [F1, K, F2] with K contiguous.
struct Layout {
  bool contiguous = false;
  int s = 0;     // first K position
  Labs korder;   // K labels in stored order
};

inline Layout classify(const Labs& lab, const Labs& K) {
  Layout L;
  if (K.n == 0) {
    L.contiguous = true;
    L.s = lab.n;
    return L;
  }
  int first = lab.n, last = -1;
  for (int p = 0; p < lab.n; ++p)
    if (K.at(lab.v[p]) >= 0) {
      first = std::min(first, p);
      last = p;
      L.korder.push_back(lab.v[p]);
    }
  L.contiguous = last - first + 1 == K.n;
  L.s = first;
  return L;
}

// How two labelled operands are contracted over their shared labels K: the order each is
// brought to first (its own when it is used in place) and the result's label order.
struct PairPlan {
  Labs K, a, b, out;
  Layout la, lb;
  bool perm_a = false, perm_b = false;
  bool batched_a() const { return la.contiguous && la.s > 0 && la.s + K.n < a.n; }
  bool batched_b() const { return lb.contiguous && lb.s > 0 && lb.s + K.n < b.n; }
};

template <typename Dim>  // dim(label): its extent
PairPlan plan_pair(const Labs& labA, double sizeA, const Labs& labB, double sizeB, Dim dim) {
  PairPlan p;
  p.a = labA;
  p.b = labB;
  for (int l : labA)
    if (labB.at(l) >= 0) p.K.push_back(l);
  p.la = classify(p.a, p.K);
  p.lb = classify(p.b, p.K);
  auto canon_A = [&](const Labs& korder) {
    Labs ord;
    for (int l : p.a)
      if (p.K.at(l) < 0) ord.push_back(l);
    ord.append(korder, 0, korder.n);
    p.a = ord;
    p.perm_a = true;
    p.la = classify(p.a, p.K);
  };
  auto canon_B = [&](const Labs& korder) {
    Labs ord = korder;
    for (int l : p.b)
      if (p.K.at(l) < 0) ord.push_back(l);
    p.b = ord;
    p.perm_b = true;
    p.lb = classify(p.b, p.K);
  };
  // Fix operands that cannot be used in place.
  if (!p.la.contiguous && !p.lb.contiguous) {
    canon_A(p.K);
    canon_B(p.la.korder);
  } else if (!p.la.contiguous) {
    canon_A(p.lb.korder);
  } else if (!p.lb.contiguous) {
    canon_B(p.la.korder);
  }
  // A batched product is as wide as the batched operand's first free labels: a site label of
  // extent 2 there leaves a tensor-core tile 2 columns (and an FP64 tile 2 of its 16).  One
  // permutation makes it wide: products 256 x 2 x 1280 by 512 of the environments took two
  // thirds of the FP64 time of a sweep (N = 22, bonds to 256: FP64 products 101 ms of four
  // sweeps, 46 with the permutation).
  auto extent = [&](const Labs& x, int from, int to) {
    double e = 1;
    for (int k = from; k < to; ++k) e *= double(dim(x.v[k]));
    return e;
  };
  auto thin = [&](const Labs& x, const Layout& L) {
    const double inner = extent(x, 0, L.s), batch = extent(x, L.s + p.K.n, x.n);
    return inner < 32 && inner * batch >= 64 && extent(p.K, 0, p.K.n) >= 64;
  };
  if (p.batched_a() && thin(p.a, p.la)) canon_A(p.lb.korder);
  if (p.batched_b() && thin(p.b, p.lb)) canon_B(p.la.korder);
  if (p.batched_a() && p.batched_b()) {
    if (sizeA <= sizeB)
      canon_A(p.lb.korder);
    else
      canon_B(p.la.korder);
  }
  if (p.la.korder != p.lb.korder) {
    // permute the smaller operand to the other's K order (unless that one is batched)
    bool permA = sizeA <= sizeB;
    if (p.batched_b()) permA = true;
    if (p.batched_a()) permA = false;
    if (permA)
      canon_A(p.lb.korder);
    else
      canon_B(p.la.korder);
  }
  const int a2 = p.la.s + p.K.n, b2 = p.lb.s + p.K.n;  // where the trailing free labels begin
  if (p.la.s > 0 && a2 < p.a.n) {
    p.out.append(p.a, 0, p.la.s);
    if (p.lb.s > 0)
      p.out.append(p.b, 0, p.lb.s);
    else
      p.out.append(p.b, b2, p.b.n);
    p.out.append(p.a, a2, p.a.n);
  } else {
    p.out.append(p.a, 0, p.la.s);
    p.out.append(p.a, a2, p.a.n);
    p.out.append(p.b, 0, p.lb.s);
    p.out.append(p.b, b2, p.b.n);
  }
  return p;
}

// ---------------------------------------------------------------------------
// contraction trees
// ---------------------------------------------------------------------------
struct Node {
  int leaf = -1;          // tensor index for leaves
  int left = -1, right = -1;
  uint32_t mask = 0;
  Labs order;              // labels of the intermediate, as contract_pair leaves them
  double size = 1;         // its elements
  double flops = 0;        // MACs of this step
};

struct Tree {
  std::vector<Node> nodes;
  int root = -1;
  double total_macs = 0;
};

// Exact flop-optimal pairwise order (dynamic programming over subsets).  Trees of equal
// flops are common (both ends of a chain's H_eff, either operand of a step first), and
// differ in the permutations that contract_pair needs: among them one that moves little
// data is taken, a permutation counting as its elements plus kPermLaunch for the launch.
// For that a subset keeps, of its flop-optimal trees, the cheapest per order of its result
// (up to kOrders of them, and none that a permutation of the cheapest would beat).  (Taking
// the first tree cost a permutation of the 168 MB intermediate per application at bond
// dimension 1024: 0.6 of 3.5 ms.)
constexpr double kPermLaunch = 2e4;
constexpr size_t kOrders = 6;

inline Tree optimal_tree(const std::vector<std::vector<int>>& labs, const std::vector<int>& out_labels,
                         const std::unordered_map<int, int64_t>& dims) {
  const int n = int(labs.size());
  NSG_CHECK(n >= 1 && n <= 12, NSG_ERR_UNSUPPORTED, "contract: 1..12 tensors");
  const uint32_t full = (1u << n) - 1;
  // labels: the tensors that hold each, its dimension, whether it is in the result
  struct Label {
    uint32_t where = 0;
    double dim = 1;
    bool out = false;
  };
  std::vector<Label> lab;
  {
    std::unordered_map<int, int> index;
    auto label_of = [&](int l) -> Label& {
      auto it = index.emplace(l, int(lab.size()));
      if (it.second) {
        lab.push_back(Label());
        lab.back().dim = double(dims.at(l));
      }
      return lab[it.first->second];
    };
    for (int i = 0; i < n; ++i)
      for (int l : labs[i]) label_of(l).where |= 1u << i;
    for (int l : out_labels) label_of(l).out = true;
  }
  auto open_in = [&](const Label& l, uint32_t S) { return (l.where & S) && ((l.where & ~S & full) || l.out); };
  struct Cand {
    double moved = 0;
    Labs order;
    uint32_t left = 0, right = 0;
    int ci = 0, cj = 0;  // the parts' candidates
  };
  struct State {
    double flops = 0, size = 1;
    std::vector<uint32_t> splits;  // of the least flops: the larger part
    std::vector<Cand> cands;
  };
  std::vector<State> st(size_t(1) << n);
  for (uint32_t S = 1; S <= full; ++S) {
    State& s = st[S];
    for (const Label& l : lab)
      if (open_in(l, S)) s.size *= l.dim;
    if ((S & (S - 1)) == 0) continue;
    s.flops = INFINITY;
    for (uint32_t S1 = (S - 1) & S; S1 > 0; S1 = (S1 - 1) & S) {
      const uint32_t S2 = S & ~S1;
      if (S1 < S2) continue;
      // multiply-adds of the step: the labels open in either part
      double f = 1;
      for (const Label& l : lab)
        if (open_in(l, S1) || open_in(l, S2)) f *= l.dim;
      f += st[S1].flops + st[S2].flops;
      if (f > s.flops * (1 + 1e-9)) continue;
      if (f < s.flops * (1 - 1e-9)) {
        s.flops = f;
        s.splits.clear();
      }
      s.splits.push_back(S1);
    }
  }
  const Labs result(out_labels);
  std::function<void(uint32_t)> plan = [&](uint32_t S) {
    State& s = st[S];
    if (!s.cands.empty()) return;
    if ((S & (S - 1)) == 0) {
      int i = 0;
      while (!((S >> i) & 1)) ++i;
      Cand leaf;
      leaf.order = Labs(labs[i]);
      s.cands.push_back(leaf);
      return;
    }
    for (uint32_t S1 : s.splits) {
      const uint32_t S2 = S & ~S1;
      plan(S1);
      plan(S2);
      for (int i = 0; i < int(st[S1].cands.size()); ++i)
        for (int j = 0; j < int(st[S2].cands.size()); ++j)
          for (int swap = 0; swap < 2; ++swap) {
            const uint32_t A = swap ? S2 : S1, B = swap ? S1 : S2;
            const Cand &ca = st[A].cands[swap ? j : i], &cb = st[B].cands[swap ? i : j];
            Cand q;
            q.moved = ca.moved + cb.moved;
            const PairPlan p = plan_pair(ca.order, st[A].size, cb.order, st[B].size, [&](int l) { return dims.at(l); });
            if (p.perm_a) q.moved += st[A].size + kPermLaunch;
            if (p.perm_b) q.moved += st[B].size + kPermLaunch;
            q.order = p.out;
            if (S == full && p.out != result) {
              // (a plain product in the swapped order is formed transposed)
              Labs t;
              t.append(p.b, 0, p.lb.s);
              t.append(p.b, p.lb.s + p.K.n, p.b.n);
              t.append(p.a, 0, p.la.s);
              t.append(p.a, p.la.s + p.K.n, p.a.n);
              if (p.batched_a() || p.batched_b() || t != result) q.moved += s.size + kPermLaunch;
              q.order = result;
            }
            q.left = A;
            q.right = B;
            q.ci = swap ? j : i;
            q.cj = swap ? i : j;
            auto same = std::find_if(s.cands.begin(), s.cands.end(), [&](const Cand& x) { return x.order == q.order; });
            if (same == s.cands.end())
              s.cands.push_back(q);
            else if (q.moved < same->moved)
              *same = q;
          }
    }
    std::stable_sort(s.cands.begin(), s.cands.end(), [](const Cand& x, const Cand& y) { return x.moved < y.moved; });
    const double most = s.cands[0].moved + s.size + kPermLaunch;
    while (s.cands.size() > kOrders || s.cands.back().moved >= most) s.cands.pop_back();
  };
  plan(full);
  Tree T;
  std::function<int(uint32_t, int)> build = [&](uint32_t S, int k) -> int {
    const Cand& q = st[S].cands[k];
    Node nd;
    nd.mask = S;
    nd.order = q.order;
    nd.size = st[S].size;
    if ((S & (S - 1)) == 0) {
      int i = 0;
      while (!((S >> i) & 1)) ++i;
      nd.leaf = i;
    } else {
      nd.left = build(q.left, q.ci);
      nd.right = build(q.right, q.cj);
      nd.flops = st[S].flops - st[q.left].flops - st[q.right].flops;
      T.total_macs += nd.flops;
    }
    T.nodes.push_back(nd);
    return int(T.nodes.size()) - 1;
  };
  T.root = build(full, 0);
  return T;
}

}  // namespace nsg
