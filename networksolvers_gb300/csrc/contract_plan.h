// Planning of tensor-network contractions (contract.cu runs the plans): how two labelled
// operands become one (strided-batched) product, and in which pairwise order a network is
// contracted.  Host code without device calls.
#pragma once

#include "nsg_internal.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <functional>
#include <iterator>
#include <unordered_map>
#include <vector>

namespace nsg {

// A short list of labels without an allocation (the planning below forms thousands).  V: int
// for the caller's labels, a byte for the search's own numbering of them.
template <typename V>
struct Labs {
  int n = 0;
  V v[2 * NSG_MAX_RANK];
  Labs() {}
  Labs(const std::vector<int>& x) {
    NSG_CHECK(x.size() <= 2 * NSG_MAX_RANK, NSG_ERR_UNSUPPORTED, "contract: result rank above 16");
    for (int l : x) push_back(V(l));
  }
  void push_back(V l) {
    NSG_CHECK(n < 2 * NSG_MAX_RANK, NSG_ERR_UNSUPPORTED, "contract: result rank above 16");
    v[n++] = l;
  }
  void append(const Labs& o, int from, int to) {
    for (int k = from; k < to; ++k) push_back(o.v[k]);
  }
  const V* begin() const { return v; }
  const V* end() const { return v + n; }
  int at(V l) const {
    for (int k = 0; k < n; ++k)
      if (v[k] == l) return k;
    return -1;
  }
  bool operator==(const Labs& o) const { return n == o.n && std::equal(v, v + n, o.v); }
  bool operator!=(const Labs& o) const { return !(*this == o); }
  std::vector<int> list() const { return std::vector<int>(v, v + n); }
};

// Where the contracted labels sit inside an operand: [F1, K, F2] with K contiguous.
template <typename V>
struct Layout {
  bool contiguous = false;
  int s = 0;       // first K position
  Labs<V> korder;  // K labels in stored order
};

template <typename V>
Layout<V> classify(const Labs<V>& lab, const Labs<V>& K) {
  Layout<V> L;
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
template <typename V>
struct PairPlan {
  Labs<V> K, a, b, out;
  Layout<V> la, lb;
  bool perm_a = false, perm_b = false;
  bool widened = false;  // a permutation that only makes a batched product wide
  bool batched_a() const { return la.contiguous && la.s > 0 && la.s + K.n < a.n; }
  bool batched_b() const { return lb.contiguous && lb.s > 0 && lb.s + K.n < b.n; }
  // rows and columns of the product, of each batch entry
  template <typename Dim>
  void free_sizes(Dim dim, double* M, double* N) const {
    auto extent = [&](const Labs<V>& x, const Layout<V>& L, bool one) {  // one: the batched operand's first group
      double e = 1;
      for (int q = 0; q < x.n; ++q)
        if (q < L.s || (q >= L.s + K.n && !one)) e *= double(dim(x.v[q]));
      return e;
    };
    *M = extent(a, la, batched_a());
    *N = extent(b, lb, batched_b());
  }
};

template <typename V, typename Dim>  // dim(label): its extent
PairPlan<V> plan_pair(const Labs<V>& labA, double sizeA, const Labs<V>& labB, double sizeB, Dim dim, bool widen = true) {
  PairPlan<V> p;
  p.a = labA;
  p.b = labB;
  for (V l : labA)
    if (labB.at(l) >= 0) p.K.push_back(l);
  p.la = classify(p.a, p.K);
  p.lb = classify(p.b, p.K);
  auto canon_A = [&](const Labs<V>& korder) {
    Labs<V> ord;
    for (V l : p.a)
      if (p.K.at(l) < 0) ord.push_back(l);
    ord.append(korder, 0, korder.n);
    p.a = ord;
    p.perm_a = true;
    p.la = classify(p.a, p.K);
  };
  auto canon_B = [&](const Labs<V>& korder) {
    Labs<V> ord = korder;
    for (V l : p.b)
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
  auto extent = [&](const Labs<V>& x, int from, int to) {
    double e = 1;
    for (int k = from; k < to; ++k) e *= double(dim(x.v[k]));
    return e;
  };
  auto thin = [&](const Labs<V>& x, const Layout<V>& L) {
    const double inner = extent(x, 0, L.s), batch = extent(x, L.s + p.K.n, x.n);
    return inner < 32 && inner * batch >= 64 && extent(p.K, 0, p.K.n) >= 64;
  };
  if (widen && p.batched_a() && thin(p.a, p.la)) {
    canon_A(p.lb.korder);
    p.widened = true;
  }
  if (widen && p.batched_b() && thin(p.b, p.lb)) {
    canon_B(p.la.korder);
    p.widened = true;
  }
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
  Labs<int> order;         // labels of the intermediate, as contract_pair leaves them
  double size = 1;         // its elements
  double flops = 0;        // MACs of this step
};

struct Tree {
  std::vector<Node> nodes;
  int root = -1;
  double total_macs = 0;
  double moved = 0;        // what its permutations cost
  double fp64_macs = 0;    // MACs of the products below the tensor-core form's sizes
};

// Exact flop-optimal pairwise order (dynamic programming over subsets) among those whose
// intermediates have no more labels than a tensor holds.  Trees of equal flops are common
// (both ends of a chain's H_eff, either operand of a step first), and differ in the
// permutations that contract_pair needs and, in the split precisions, in the products that
// miss the tensor-core form's least sizes.  Among them one of little predicted time is taken,
// in units of an element's permutation (16 bytes of HBM traffic, 2.4 ps; twice both for
// complex data): a permutation costs its elements plus kPermLaunch, a multiply-add 0.7 on the
// FP64 cores (two per clock and SM) and 0.02 as a split product (4096 x 1024 x 1024 in 0.17
// ms), twice those for complex data, whose elements take two and whose multiply-adds four
// times as long; a split product costs kSplitLaunch beyond that (an eigensolve with bonds 40 and
// 100 takes 376 us with the 3.2 million multiply-adds of one product of its H_eff on the FP64
// cores and 400 with them split; 63 and 100, 7.9 million: 426 and 415).  For that a subset
// keeps, of its flop-optimal trees, the cheapest per order of its result (none that a
// permutation of the cheapest would beat).  Taking the first tree cost a permutation of the
// 168 MB intermediate per application at bond dimension 1024, 0.6 of 3.5 ms; counting
// permutations alone left 25 % of the multiply-adds of an H_eff with bonds 60 and 240 to the
// FP64 cores and 45 % with bonds 63 and 100, where 6 % and 11 % need be (eigensolves with bonds
// 60 and 240: 543 us and 482; 60 and 1000: 551 and 470).
//
// Where bonds are equal, or 1 as in a product state, almost every tree ties.  The search is
// cut to a number of pair plans that takes no longer than the dynamic programming itself:
// fewer splits per subset, and fewer orders, the more trees tie.  Planning times, host of the
// GPU machine's class: H_eff of a chain 8 us, environment at a vertex of degree 6 0.3 ms, twelve
// tensors with bonds 1 7 ms; without the limit 13 us, 3.7 ms, 6 s as a chain and 56 s as a star.
constexpr double kPermLaunch = 2e4, kSplitLaunch = 4e6;
struct SearchLimit {
  int splits, orders;
};
constexpr SearchLimit kSearch[] = {{1 << 12, 6}, {4, 6}, {3, 3}, {2, 2}, {1, 1}};

inline Tree optimal_tree(const std::vector<std::vector<int>>& labs, const std::vector<int>& out_labels,
                         const std::unordered_map<int, int64_t>& dims, int precision = NSG_PREC_FP64,
                         int dtype = NSG_F64) {
  using L = Labs<uint8_t>;
  const int n = int(labs.size());
  NSG_CHECK(n >= 1 && n <= 12, NSG_ERR_UNSUPPORTED, "contract: 1..12 tensors");
  const uint32_t full = (1u << n) - 1;
  // labels, numbered: the tensors that hold each, its dimension, whether it is in the result
  struct Label {
    int name;
    uint32_t where = 0;
    double dim = 1;
    bool out = false;
  };
  std::vector<Label> lab;
  std::vector<L> of(n);
  L result;
  {
    std::unordered_map<int, int> index;
    auto number = [&](int l) {
      auto it = index.emplace(l, int(lab.size()));
      if (it.second) lab.push_back(Label{l, 0, double(dims.at(l)), false});
      return it.first->second;  // (12 tensors of 16 labels and 16 of the result at most)
    };
    for (int i = 0; i < n; ++i)
      for (int l : labs[i]) {
        const int k = number(l);
        lab[k].where |= 1u << i;
        of[i].push_back(uint8_t(k));
      }
    for (int l : out_labels) {
      const int k = number(l);
      lab[k].out = true;
      result.push_back(uint8_t(k));
    }
  }
  auto dim = [&](uint8_t l) { return lab[l].dim; };
  // labels open in a subset, as a bit set
  constexpr int kWords = 4;
  const int words = int(lab.size() + 63) / 64;
  struct Set {
    uint64_t w[kWords] = {};
  };
  auto extent = [&](const Set& a, const Set& b) {  // of the union
    double e = 1;
    for (int k = 0; k < words; ++k)
      for (uint64_t m = a.w[k] | b.w[k]; m; m &= m - 1) e *= lab[64 * k + __builtin_ctzll(m)].dim;
    return e;
  };
  struct Cand {
    double cost = 0, moved = 0, fp64 = 0;
    L order;
    uint32_t left = 0, right = 0;
    int ci = 0, cj = 0;  // the parts' candidates
  };
  struct State {
    double flops = 0, size = 1;
    Set open;
    std::vector<uint32_t> splits;  // of the least flops: the larger part
    std::vector<Cand> cands;
    int reached = 0;  // by the limit numbered so
  };
  std::vector<State> st(size_t(1) << n);
  for (uint32_t S = 1; S <= full; ++S) {
    State& s = st[S];
    for (size_t l = 0; l < lab.size(); ++l)
      if ((lab[l].where & S) && ((lab[l].where & ~S & full) || lab[l].out)) s.open.w[l / 64] |= uint64_t(1) << (l % 64);
    s.size = extent(s.open, s.open);
    if ((S & (S - 1)) == 0) continue;
    s.flops = INFINITY;
    int rank = 0;
    for (int k = 0; k < words; ++k) rank += __builtin_popcountll(s.open.w[k]);
    if (rank > NSG_MAX_RANK) continue;
    for (uint32_t S1 = (S - 1) & S; S1 > 0; S1 = (S1 - 1) & S) {
      const uint32_t S2 = S & ~S1;
      if (S1 < S2) break;  // (descending: the rest are the mirrored splits)
      // multiply-adds of the step: the labels open in either part
      const double f = extent(st[S1].open, st[S2].open) + st[S1].flops + st[S2].flops;
      if (f == INFINITY || f > s.flops * (1 + 1e-9)) continue;
      if (f < s.flops * (1 - 1e-9)) {
        s.flops = f;
        s.splits.clear();
      }
      s.splits.push_back(S1);
    }
  }
  NSG_CHECK(st[full].flops < INFINITY, NSG_ERR_UNSUPPORTED, "contract: result rank above 16");
  auto single = [](uint32_t S) { return (S & (S - 1)) == 0; };
  // pair plans that a limit takes at most, over the subsets below S not yet counted
  std::function<double(uint32_t, SearchLimit, int)> pairs = [&](uint32_t S, SearchLimit lim, int mark) -> double {
    if (single(S) || st[S].reached == mark) return 0.0;
    st[S].reached = mark;
    double c = 0;
    for (int k = 0; k < std::min(lim.splits, int(st[S].splits.size())); ++k) {
      const uint32_t S1 = st[S].splits[k], S2 = S & ~S1;
      c += 2.0 * (single(S1) ? 1 : lim.orders) * (single(S2) ? 1 : lim.orders);
      c += pairs(S1, lim, mark) + pairs(S2, lim, mark);
    }
    return c;
  };
  if (precision == NSG_PREC_TF32X3 && dtype == NSG_C128) precision = NSG_PREC_FP64;  // (real data only)
  const double mac_scale = dtype == NSG_C128 ? 2.0 : 1.0;
  SearchLimit lim = kSearch[0];
  for (int k = 0; k < int(std::size(kSearch)); ++k) {
    lim = kSearch[k];
    if (pairs(full, lim, k + 1) <= std::max(200.0, std::min(std::pow(3.0, n) / 4, 2e4))) break;
  }
  std::function<void(uint32_t)> plan = [&](uint32_t S) {
    State& s = st[S];
    if (!s.cands.empty()) return;
    if (single(S)) {
      Cand leaf;
      leaf.order = of[__builtin_ctz(S)];
      s.cands.push_back(leaf);
      return;
    }
    for (int k = 0; k < std::min(lim.splits, int(s.splits.size())); ++k) {
      const uint32_t S1 = s.splits[k], S2 = S & ~S1;
      plan(S1);
      plan(S2);
      for (int i = 0; i < int(st[S1].cands.size()); ++i)
        for (int j = 0; j < int(st[S2].cands.size()); ++j)
          for (int swap = 0; swap < 2; ++swap) {
            const uint32_t A = swap ? S2 : S1, B = swap ? S1 : S2;
            const Cand &ca = st[A].cands[swap ? j : i], &cb = st[B].cands[swap ? i : j];
            Cand q;
            const auto p = plan_pair(ca.order, st[A].size, cb.order, st[B].size, dim);
            double moved = 0;
            if (p.perm_a) moved += st[A].size + kPermLaunch;
            if (p.perm_b) moved += st[B].size + kPermLaunch;
            q.order = p.out;
            bool transposed = false;
            if (S == full && p.out != result) {
              // (a plain product in the swapped order is formed transposed)
              L t;
              t.append(p.b, 0, p.lb.s);
              t.append(p.b, p.lb.s + p.K.n, p.b.n);
              t.append(p.a, 0, p.la.s);
              t.append(p.a, p.la.s + p.K.n, p.a.n);
              transposed = !p.batched_a() && !p.batched_b() && t == result;
              if (!transposed) moved += s.size + kPermLaunch;
              q.order = result;
            }
            double time = 0, slow = 0;
            if (precision != NSG_PREC_FP64) {
              const double macs = s.flops - st[A].flops - st[B].flops;
              double M, N, K = 1;
              p.free_sizes(dim, &M, &N);
              for (uint8_t l : p.K) K *= dim(l);
              if (transposed) std::swap(M, N);
              if (tensor_core_sizes(precision, M, N, K))
                time = kSplitLaunch + 0.02 * mac_scale * macs;
              else
                time = 0.7 * mac_scale * (slow = macs);
            }
            q.cost = ca.cost + cb.cost + moved + time;
            q.moved = ca.moved + cb.moved + moved;
            q.fp64 = ca.fp64 + cb.fp64 + slow;
            q.left = A;
            q.right = B;
            q.ci = swap ? j : i;
            q.cj = swap ? i : j;
            auto same = std::find_if(s.cands.begin(), s.cands.end(), [&](const Cand& x) { return x.order == q.order; });
            if (same == s.cands.end())
              s.cands.push_back(q);
            else if (q.cost < same->cost)
              *same = q;
          }
    }
    std::stable_sort(s.cands.begin(), s.cands.end(), [](const Cand& x, const Cand& y) { return x.cost < y.cost; });
    const double most = s.cands[0].cost + s.size + kPermLaunch;
    while (s.cands.size() > size_t(lim.orders) || s.cands.back().cost >= most) s.cands.pop_back();
  };
  plan(full);
  Tree T;
  std::function<int(uint32_t, int)> build = [&](uint32_t S, int k) -> int {
    const Cand& q = st[S].cands[k];
    Node nd;
    nd.mask = S;
    for (uint8_t l : q.order) nd.order.push_back(lab[l].name);
    nd.size = st[S].size;
    if (single(S)) {
      nd.leaf = __builtin_ctz(S);
    } else {
      nd.left = build(q.left, q.ci);
      nd.right = build(q.right, q.cj);
      nd.flops = st[S].flops - st[q.left].flops - st[q.right].flops;
      T.total_macs += nd.flops;
    }
    T.nodes.push_back(nd);
    return int(T.nodes.size()) - 1;
  };
  T.moved = st[full].cands[0].moved;
  T.fp64_macs = st[full].cands[0].fp64;
  T.root = build(full, 0);
  return T;
}

}  // namespace nsg
