// cdt_flips_host.cpp -- one flip round of the constrained Delaunay stage after the
// other on the CPU (csrc/cdt_core.cuh), for tests/test_cdt_flips.py: every flip that
// lost a claim reads the triangles it claimed (flip_claims) again after each winner's
// flip, as its thread on the GPU may at any time of the round.
//
// argv: N seed.  N points of a parabola, triangulated as a fan: every triangle has a
// hull edge, and flips move hull edges into the losers' triangles.
// stdout: "ok ROUNDS HULL" (HULL: reads by losers whose edge had become a hull edge),
// or "error <what>".
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "cdt_core.cuh"

using namespace cvtgb::cdt;

int main(int argc, char **argv) {
  const int N = argc > 1 ? atoi(argv[1]) : 40;
  unsigned state = argc > 2 ? (unsigned)atoi(argv[2]) : 1u;
  std::vector<i64> X(N), Y(N), R(N);
  i64 x = -(i64)N * 20;
  for (int v = 0; v < N; ++v) {
    state = state * 1664525u + 1013904223u;
    x += 1 + (state >> 24) % 40;
    X[v] = x, Y[v] = x * x, R[v] = v;
  }
  const int T = N - 2;
  std::vector<int> tri(3 * (size_t)T), nbr(3 * (size_t)T, kNone), vt(N, 0);
  std::vector<unsigned> cons(T, 0);
  for (int t = 0; t < T; ++t) {  // (0, t + 1, t + 2): counter-clockwise
    tri[3 * t] = 0, tri[3 * t + 1] = t + 1, tri[3 * t + 2] = t + 2;
    if (t + 1 < T) nbr[3 * t + 1] = pack_nb(t + 1, 2);
    if (t > 0) nbr[3 * t + 2] = pack_nb(t - 1, 1);
    vt[t + 1] = vt[t + 2] = t;
  }
  Mesh m{tri.data(), nbr.data(), cons.data(), vt.data(), X.data(), Y.data(), R.data()};
  long hull = 0;
  for (int round = 0;; ++round) {
    if (round > 100000) return printf("error rounds\n"), 0;
    std::vector<int> edge(T, -1);
    std::vector<unsigned> cl(T, 0xffffffffu);
    bool any = false;
    int id[8];
    for (int t = 0; t < T; ++t) {
      const int i = edge[t] = first_flip(m, t) - 1;
      if (i < 0) continue;
      any = true;
      flip_claims(m, t, i, id);
      for (int k : id) cl[k] = std::min(cl[k], prio((unsigned)(3 * t + i)));
    }
    if (!any) {  // Delaunay: no edge of any triangle wants a flip
      for (int t = 0; t < T; ++t)
        for (int i = 0; i < 3; ++i)
          if (wants_flip(m, t, i)) return printf("error left\n"), 0;
      return printf("ok %d %ld\n", round, hull), 0;
    }
    std::vector<int> won, lost;
    // (-1: an index out of range)
    auto owns = [&](int t) -> int {
      flip_claims(m, t, edge[t], id);
      int own = 1;
      for (int k : id) {
        if (k < 0 || k >= T) return -1;
        own &= cl[k] == prio((unsigned)(3 * t + edge[t]));
      }
      return own;
    };
    for (int t = 0; t < T; ++t)
      if (edge[t] >= 0) (owns(t) ? won : lost).push_back(t);
    if (won.empty()) return printf("error no winner\n"), 0;
    for (size_t w = 0; w < won.size(); ++w) {
      if (owns(won[w]) != 1) return printf("error winner\n"), 0;
      flip(m, won[w], edge[won[w]]);
      for (int t : lost) {
        hull += nbr[3 * t + edge[t]] < 0;
        const int own = owns(t);
        if (own < 0) return printf("error range\n"), 0;
        if (own) return printf("error loser\n"), 0;
      }
    }
  }
}
