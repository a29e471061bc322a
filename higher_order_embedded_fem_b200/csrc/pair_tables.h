// Tables over the node pairs of an element, built by the compiler: constant memory
// holds them from the start, for every stream, thread and device.  Without CUDA
// types, so that they can be checked on the CPU.
#pragma once

#ifdef __CUDACC__
#define HOEFEM_TABLE_HD __host__ __device__
#else
#define HOEFEM_TABLE_HD
#endif

namespace hoefem {

// Node pairs I >= J of an element, by columns: row node I, column node J of pair p.
template <int NN>
struct PairTable {
  static constexpr int NP = NN * (NN + 1) / 2;
  unsigned char at[NP][2];
};

template <int NN>
constexpr PairTable<NN> pair_table() {
  PairTable<NN> t{};
  int p = 0;
  for (int J = 0; J < NN; ++J)
    for (int I = J; I < NN; ++I, ++p) {
      t.at[p][0] = (unsigned char)I;
      t.at[p][1] = (unsigned char)J;
    }
  return t;
}

// Place of a symmetric 4 x 4 index pair: 00 01 02 03 11 12 13 22 23 33.
HOEFEM_TABLE_HD constexpr int sym4(int x, int y) {
  const int lo = x < y ? x : y, hi = x < y ? y : x;
  return 4 * lo - lo * (lo - 1) / 2 + hi - lo;
}

// The stiffness blocks of a Tet10 element from the moments of its tangent
// (stiffness_moments.cu).  Weights: l_v l_w at sym4(v, w), l_v at 10 + v, 1 at 14; a
// weight's ten 3 x 3 blocks of l-gradient pairs (x, y) at 9 sym4(x, y), 90 values in
// all.  Four terms per node pair: the offset of the block's first value, bit 11 set
// if it is read transposed, and the coefficient + 8 above bit 12 (16 is stored as 7).
struct MomentTerms {
  int at[55][4];
};

constexpr int moment_term(int weight, int x, int y, int coefficient) {
  return (weight * 90 + 9 * sym4(x, y)) | (x > y ? 2048 : 0) | (((coefficient == 16 ? 7 : coefficient) + 8) << 12);
}

constexpr MomentTerms moment_terms() {
  MomentTerms t{};
  const int edge[6][2] = {{0, 1}, {1, 2}, {0, 2}, {0, 3}, {2, 3}, {1, 3}};
  int p = 0;
  for (int J = 0; J < 10; ++J)
    for (int I = J; I < 10; ++I, ++p) {
      if (I < 4) {  // (4 l_I - 1) (4 l_J - 1)
        t.at[p][0] = moment_term(sym4(I, J), I, J, 16);
        t.at[p][1] = moment_term(10 + I, I, J, -4);
        t.at[p][2] = moment_term(10 + J, I, J, -4);
        t.at[p][3] = moment_term(14, I, J, 1);
        continue;
      }
      const int a = edge[I - 4][0], d = edge[I - 4][1];
      if (J < 4) {  // 4 (l_d g_a + l_a g_d), (4 l_J - 1) g_J
        t.at[p][0] = moment_term(sym4(d, J), a, J, 16);
        t.at[p][1] = moment_term(10 + d, a, J, -4);
        t.at[p][2] = moment_term(sym4(a, J), d, J, 16);
        t.at[p][3] = moment_term(10 + a, d, J, -4);
      } else {
        const int f = edge[J - 4][0], h = edge[J - 4][1];
        t.at[p][0] = moment_term(sym4(d, h), a, f, 16);
        t.at[p][1] = moment_term(sym4(d, f), a, h, 16);
        t.at[p][2] = moment_term(sym4(a, h), d, f, 16);
        t.at[p][3] = moment_term(sym4(a, f), d, h, 16);
      }
    }
  return t;
}

}  // namespace hoefem
