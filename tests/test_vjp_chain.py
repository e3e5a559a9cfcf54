"""The order of an adjoint's contraction (host code, compiled by itself): the chain of least modelled
time against all chains, the greedy one where searching is not worth its time, and that time."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graft.jl_gb300", "csrc")

PROGRAM = r"""
#include "gtn_vjp_chain.h"
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>

static double steps(double M, double K, double N) { return 14e-6 + 8 * M * K * N / 4e13 + (M * K + M * N) * 16 / 5e12; }

struct Net {
  std::vector<std::vector<std::pair<int, int64_t>>> op;  // (label, dim) legs
  double time(const std::vector<int>& ord) const {       // of a chain, from the legs themselves
    auto cur = op[ord[0]];
    double t = 0;
    for (size_t i = 1; i < ord.size(); ++i) {
      const auto& q = op[ord[i]];
      double M = 1, K = 1, N = 1;
      decltype(cur) next;
      auto has = [](const decltype(cur)& v, int l) {
        return l > 0 && std::any_of(v.begin(), v.end(), [l](const std::pair<int, int64_t>& x) { return x.first == l; });
      };
      for (auto& l : q) if (!has(cur, l.first)) { N *= l.second; next.push_back(l); }
      for (auto& l : cur) if (has(q, l.first)) K *= l.second; else { M *= l.second; next.push_back(l); }
      t += steps(M, K, N);
      cur = next;
    }
    return t;
  }
  std::vector<int> order(bool greedy) const {
    std::vector<int> r, l;
    std::vector<int64_t> d;
    for (auto& o : op) {
      r.push_back((int)o.size());
      for (auto& x : o) { l.push_back(x.first); d.push_back(x.second); }
    }
    const VjpNetwork net((int)op.size(), r, d, l);
    const auto g = net.greedy_chain();
    return greedy ? g : net.cheapest_chain(g, steps);
  }
};

// A site tensor's adjoint: cotangent, operator and nb environments; dim of every bond.
static Net site(int nb, int64_t bond, int64_t w) {
  Net n;
  n.op.resize(nb + 2);
  for (int i = 0; i < nb; ++i) {
    n.op[0].push_back({i + 1, bond});                               // cotangent: bra legs
    n.op[1].push_back({100 + i, w});                                // operator
    n.op[2 + i] = {{-(i + 1), bond}, {100 + i, w}, {i + 1, bond}};  // environments
  }
  n.op[0].push_back({200, 2});
  n.op[1].push_back({200, 2});
  n.op[1].push_back({-(nb + 1), 2});
  return n;
}

int main() {
  std::mt19937 rng(1);
  int searched = 0;
  for (int it = 0; it < 400; ++it) {
    const int n = 3 + (int)(rng() % 4);
    Net net;
    net.op.resize(n);
    int lab = 0, out = 0;
    const double big = it % 2 ? 6.0 : 3.0;
    auto dim = [&] { return (int64_t)std::lround(std::pow(2.0, big * (rng() % 1000) / 1000.0)); };
    for (int e = 0; e < n + 3; ++e) {
      const int i = (int)(rng() % n), j = (int)(rng() % n);
      if (i == j) continue;
      const int64_t d = dim();
      net.op[i].push_back({++lab, d});
      net.op[j].push_back({lab, d});
    }
    for (int i = 0; i < n; ++i)
      if (rng() % 2) net.op[i].push_back({-++out, dim()});
    const auto got = net.order(false), greedy = net.order(true);
    std::vector<int> ord(n);
    for (int i = 0; i < n; ++i) ord[i] = i;
    auto sorted = got;
    std::sort(sorted.begin(), sorted.end());
    if (sorted != ord || got[0] != 0) return 1;
    // all chains that take an outer product only where nothing connects
    double best = 1e30;
    do {
      bool ok = ord[0] == 0;
      std::vector<int> in(1, 0);
      for (int s = 1; s < n && ok; ++s) {
        auto meets = [&](int q) {
          for (int i : in)
            for (auto& x : net.op[i])
              for (auto& y : net.op[q])
                if (x.first > 0 && x.first == y.first) return true;
          return false;
        };
        if (!meets(ord[s]))
          for (int q = 1; q < n; ++q)
            if (std::find(in.begin(), in.end(), q) == in.end() && meets(q)) ok = false;
        in.push_back(ord[s]);
      }
      if (ok) best = std::min(best, net.time(ord));
    } while (std::next_permutation(ord.begin(), ord.end()));
    const double t = net.time(got), tg = net.time(greedy);
    const double pairs = (double)(1 << (n - 1)) * (n - 1) / 2;
    if (tg - (n - 1) * steps(1, 1, 1) >= pairs * kVjpPairSeconds) {
      ++searched;
      if (t > best * (1 + 1e-12)) return 2;  // the search finds the best
    } else if (got != greedy) {
      return 3;
    }
    if (t > tg * (1 + 1e-12)) return 4;
  }
  if (searched < 50) return 5;
  // the host time of networks of up to 13 operands and of more
  for (int nb : {3, 5, 9, 11, 12, 20}) {
    const Net small = site(nb, 2, 2), large = nb < 6 ? site(nb, 64, 5) : site(nb, 4, 3);
    for (const Net* n : {&small, &large}) {
      double best = 1e9;
      for (int r = 0; r < 5; ++r) {
        const auto t0 = std::chrono::steady_clock::now();
        n->order(false);
        best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
      }
      const double t = n->time(n->order(true));
      std::printf("%d operands: %.1f us of %.0f us\n", nb + 2, best * 1e6, t * 1e6);
      // on small bonds next to nothing (the exhaustive search took 12 ms at 13 operands); else at most
      // what the greedy chain may lose, with a margin for slow machines
      if (n == &small && best > 300e-6) return 6;
      if (n == &large && best > 300e-6 + 3 * t) return 7;
    }
  }
  return 0;
}
"""


def test_chain_search(tmp_path):
    src = tmp_path / "chain.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "chain"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, (r.returncode, r.stdout)
