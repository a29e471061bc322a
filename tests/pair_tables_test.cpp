// Checks csrc/pair_tables.h: the node pairs' order, and the Tet10 terms by the
// identity they stand for, K_IJ = A(grad N_I, grad N_J) at single points.
#include "pair_tables.h"

#include <cmath>
#include <cstdio>
#include <random>

using namespace hoefem;

static constexpr PairTable<10> p10 = pair_table<10>();
static constexpr PairTable<27> p27 = pair_table<27>();
static constexpr MomentTerms terms = moment_terms();

template <int NN>
static bool pairs_ok(const PairTable<NN>& t) {
  for (int p = 0; p < PairTable<NN>::NP; ++p) {
    const int I = t.at[p][0], J = t.at[p][1];
    if (J > I || I >= NN || J * NN - J * (J - 1) / 2 + I - J != p) return false;
  }
  return true;
}

int main() {
  if (!pairs_ok(p10) || !pairs_ok(p27)) {
    std::printf("pairs\n");
    return 1;
  }
  std::mt19937 rng(1);
  std::normal_distribution<double> nd;
  for (int rep = 0; rep < 20; ++rep) {
    double l[4], g[4][3], C[9][9], A4[4][4][3][3];
    double sum = 0.0;
    for (int v = 0; v < 3; ++v) sum += l[v] = 0.25 * nd(rng);
    l[3] = 1.0 - sum;
    for (int k = 0; k < 3; ++k) {
      g[0][k] = 0.0;
      for (int v = 1; v < 4; ++v) g[0][k] -= g[v][k] = nd(rng);
    }
    // a form with the tangent's symmetry, A(a, b)[i][j] = A(b, a)[j][i]
    for (int r = 0; r < 9; ++r)
      for (int c = 0; c <= r; ++c) C[r][c] = C[c][r] = nd(rng);
    auto form = [&](const double* a, const double* b, int i, int j) {
      double s = 0.0;
      for (int k = 0; k < 3; ++k)
        for (int m = 0; m < 3; ++m) s += C[3 * i + k][3 * j + m] * a[k] * b[m];
      return s;
    };
    for (int x = 0; x < 4; ++x)
      for (int y = 0; y < 4; ++y)
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) A4[x][y][i][j] = form(g[x], g[y], i, j);
    // the moments of one point
    double B[15 * 90];
    for (int w = 0; w < 15; ++w) {
      double lw = w == 14 ? 1.0 : (w >= 10 ? l[w - 10] : 0.0);
      for (int v = 0; v < 4 && w < 10; ++v)
        for (int z = v; z < 4; ++z)
          if (sym4(v, z) == w) lw = l[v] * l[z];
      for (int x = 0; x < 4; ++x)
        for (int y = x; y < 4; ++y)
          for (int k = 0; k < 9; ++k) B[90 * w + 9 * sym4(x, y) + k] = lw * A4[x][y][k / 3][k % 3];
    }
    // gradients of the quadratic functions, node order: vertices, then edges
    static const int edge[6][2] = {{0, 1}, {1, 2}, {0, 2}, {0, 3}, {2, 3}, {1, 3}};
    double G[10][3];
    for (int k = 0; k < 3; ++k) {
      for (int v = 0; v < 4; ++v) G[v][k] = (4.0 * l[v] - 1.0) * g[v][k];
      for (int e = 0; e < 6; ++e)
        G[4 + e][k] = 4.0 * (l[edge[e][1]] * g[edge[e][0]][k] + l[edge[e][0]] * g[edge[e][1]][k]);
    }
    for (int p = 0; p < 55; ++p)
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
          double s = 0.0, size = 0.0;
          for (int n = 0; n < 4; ++n) {
            const int c = terms.at[p][n], k = (c >> 12) - 8, at = c & 2047;
            const double t = (k == 7 ? 16 : k) * B[at + (c & 2048 ? 3 * j + i : 3 * i + j)];
            s += t;
            size += std::fabs(t);
          }
          const double want = form(G[p10.at[p][0]], G[p10.at[p][1]], i, j);
          if (!(std::fabs(s - want) <= 1e-12 * (1.0 + size))) {
            std::printf("terms of pair %d: %g %g\n", p, s, want);
            return 1;
          }
        }
  }
  std::printf("ok\n");
  return 0;
}
