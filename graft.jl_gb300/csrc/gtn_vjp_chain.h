// Order of contraction of an adjoint: the rewritten network (operand 0 = the cotangent) and its chains
// from operand 0.  Host code without CUDA.
#pragma once
#include <cstddef>
#include <cstdint>
#include <map>
#include <vector>

constexpr int kVjpSearchMax = 13;  // operands up to which every left-deep chain is compared
// Seconds of the search for each pair of a partial chain and a next operand.  It runs on the host in
// every call, so it has to be paid for by what the greedy chain could lose at most.
constexpr double kVjpPairSeconds = 1e-7;

class VjpNetwork {
 public:
  VjpNetwork(int n, const std::vector<int>& ranks, const std::vector<int64_t>& dims, const std::vector<int>& labels)
      : n_(n), all_(n, 1.0), bonds_(n) {
    std::map<int, int> first;  // label -> the operand that had it
    size_t o = 0;
    for (int i = 0; i < n; ++i)
      for (int r = 0; r < ranks[i]; ++r, ++o) {
        all_[i] *= (double)dims[o];
        if (labels[o] <= 0) continue;
        const auto it = first.insert({labels[o], i}).first;
        if (it->second == i) continue;
        add_bond(i, it->second, (double)dims[o]);
        add_bond(it->second, i, (double)dims[o]);
      }
  }

  // Always the operand sharing the largest contracted extent (ties: the smaller result).
  std::vector<int> greedy_chain() const {
    std::vector<int> ord(1, 0);
    std::vector<bool> in(n_, false);
    in[0] = true;
    double size = all_[0];
    for (int step = 1; step < n_; ++step) {
      int best = -1;
      double best_shared = 0, best_size = 0;
      for (int q = 1; q < n_; ++q) {
        if (in[q]) continue;
        double M, K, N;
        const double shared = absorb(size, q, [&](int i) { return in[i]; }, &M, &K, &N) ? K : 0;
        if (best < 0 || shared > best_shared || (shared == best_shared && M * N < best_size)) {
          best = q;
          best_shared = shared;
          best_size = M * N;
        }
      }
      size = best_size;
      in[best] = true;
      ord.push_back(best);
    }
    return ord;
  }

  // The chain of least modelled time (step_time(M, K, N) of absorbing an operand), or the greedy one
  // where that is as good, the network too large, or the search not worth its time.  The size of a
  // partial chain depends only on the set of its operands, so the best way to every set is built from
  // the sets with one operand less; those that cannot beat the greedy chain, with every further step as
  // short as the shortest there is, are left out.  The greedy chain takes up to five times the
  // multiply-adds: site and operator adjoints of a degree-3 node at bond 75, 50.2 -> 3.24 ms.
  template <class F> std::vector<int> cheapest_chain(const std::vector<int>& greedy, F step_time) const {
    const int n = n_ - 1;
    if (n_ > kVjpSearchMax || n < 2) return greedy;
    const double shortest = step_time(1.0, 1.0, 1.0);
    double bound = 0, size = all_[0];
    uint32_t set = 1;
    for (int i = 1; i < n_; ++i) {
      double M, K, N;
      absorb(size, greedy[i], [set](int j) { return set >> j & 1u; }, &M, &K, &N);
      bound += step_time(M, K, N);
      size = M * N;
      set |= 1u << greedy[i];
    }
    const double pairs = (double)(size_t(1) << n) * n / 2;
    if (bound - n * shortest < pairs * kVjpPairSeconds) return greedy;
    struct State {
      double cost = -1, size = 0;
      int last = -1;
    };
    std::vector<State> st(size_t(1) << n);
    st[0].cost = 0;
    st[0].size = all_[0];
    for (uint32_t mask = 0; mask + 1 < (1u << n); ++mask) {
      if (st[mask].cost < 0) continue;
      const uint32_t from = mask << 1 | 1u;
      const int left = n - __builtin_popcount(mask) - 1;  // steps after the next
      for (int pass = 0, found = 0; pass < 2 && !found; ++pass)  // outer products only if nothing connects
        for (int b = 0; b < n; ++b) {
          if (mask >> b & 1u) continue;
          double M, K, N;
          if (!absorb(st[mask].size, b + 1, [from](int j) { return from >> j & 1u; }, &M, &K, &N) && pass == 0) continue;
          found = 1;
          State& t = st[mask | 1u << b];
          const double c = st[mask].cost + step_time(M, K, N);
          if (c + left * shortest < bound && (t.cost < 0 || c < t.cost)) {
            t.cost = c;
            t.size = M * N;
            t.last = b;
          }
        }
    }
    uint32_t mask = (1u << n) - 1;
    if (st[mask].cost < 0) return greedy;  // nothing beats it
    std::vector<int> ord(n + 1, 0);
    for (int i = n; mask; --i) {
      ord[i] = st[mask].last + 1;
      mask &= ~(1u << st[mask].last);
    }
    return ord;
  }

 private:
  struct Bond {
    int other;
    double dim;  // product of the legs that two operands share
  };
  void add_bond(int i, int j, double d) {
    for (Bond& b : bonds_[i])
      if (b.other == j) {
        b.dim *= d;
        return;
      }
    bonds_[i].push_back(Bond{j, d});
  }
  // Absorb operand q into the partial chain of `size` elements over the operands in(i): the step's
  // (M, K, N), and whether they share a leg.
  template <class In> bool absorb(double size, int q, In in, double* M, double* K, double* N) const {
    bool shared = false;
    *K = 1;
    for (const Bond& b : bonds_[q])
      if (in(b.other)) {
        *K *= b.dim;
        shared = true;
      }
    *M = size / *K;
    *N = all_[q] / *K;
    return shared;
  }

  int n_;
  std::vector<double> all_;  // elements of the operands
  std::vector<std::vector<Bond>> bonds_;
};
