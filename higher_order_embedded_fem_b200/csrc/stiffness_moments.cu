// FP64 element stiffness of Tet10 blocks with one quadrature rule, from moments
// of the tangent.
//
// Reference: fenris/src/assembly.rs:746-797 (element stiffness),
// fenris/src/solid/materials.rs:689-743 (stress contraction).
//
// A Tet10 gradient is linear in the barycentric functions l_v: with g_v the
// (constant) gradient of l_v, grad N_I = (4 l_I - 1) g_I for a vertex and
// grad N_(a,b) = 4 (l_b g_a + l_a g_b) for the node of an edge.  The stiffness
// block is bilinear in the two gradients, so every K_IJ is a combination of at
// most four blocks
//   M^{vw}_{xy} = sum_q W_q l_v l_w A_q(g_x, g_y),  A_q(a, b) the 3 x 3 contraction
// and of the same with weights l_v and 1.  g_0 = -(g_1 + g_2 + g_3) leaves six
// blocks A_q(g_x, g_y) per point (45 numbers, the diagonal ones symmetric), and
// 15 weighted sums of them over the points.  Per element of the 14-point rule
// 14 x (560 + 45 x 15) + 3,000 operations instead of 55 x 14 x 62, and the pair
// loop's operands are no longer read from shared memory per pair (31
// loads for 60 FMAs, which bound it).  201,600 elements: 2.56 -> 0.81 ms (0.8 GB
// of blocks written).  Bound by shared memory, whose pipe is at 78 % of its peak
// (FP64 34 %): phase B reads 45 values and a weight for 45 FMAs, and the eight
// warps per SM that fit do not hide the rest.
// Relative error against extended precision 3.1e-16 to 3.9e-16 (boxes of 216 and
// 1,080 elements) where the pair loop has 2.1e-16 to 2.7e-16: the four terms of a
// pair cancel in part, so the rounding of the moments' sums counts more.
//
// Taken for every uniform Tet10 rule in the staged path; the pair loop
// (k_stiffness) keeps the FP32 blocks, per-element rules, the colored scatter and
// the dense element matrices of the projection.
//
// 16 threads per element, EPC elements per CTA:
//  A  thread = point: F, material state, the six blocks, into shared memory
//  B  thread = weight (15): 45 sums over the points in registers (the 16
//     threads of an element read the same operands), then the four blocks that
//     involve g_0, all ten into shared memory
//  C  the 55 x 9 values of the element's node pairs, consecutive threads to
//     consecutive addresses, from a table of four terms per pair
#include <cuda_runtime.h>

#include "element_math.cuh"
#include "internal.h"
#include "pair_tables.h"

namespace hoefem {

namespace {

constexpr int EPC = 8;           // elements per CTA
constexpr int TPE = 16;          // threads per element
constexpr int QT = 16;           // points per tile
constexpr int NW = 15;           // weights: l_v l_w (10), l_v (4), 1
constexpr int AS = 46;           // doubles per point (45, even)
constexpr int ASE = QT * AS + 2;     // per element: the two elements of a warp on different banks
constexpr int BSE = NW * 90 + 2;
constexpr int NPAIR = 55;

__constant__ MomentTerms c_terms = moment_terms();

__global__ void __launch_bounds__(EPC* TPE, 2) k_stiffness_moments(const BlockDev b, const double* __restrict__ X,
                                                                   const double* __restrict__ u,
                                                                   const double* __restrict__ weights, MatDev mat,
                                                                   int* err, double* __restrict__ pblk) {
  extern __shared__ __align__(16) double smem[];
  __shared__ double s_u[EPC][30], s_x[EPC][12];
  __shared__ double s_w[QT][16];
  __shared__ int s_ok[EPC];
  const int el = threadIdx.x / TPE, sub = threadIdx.x % TPE;
  const int e = blockIdx.x * EPC + el;
  const bool active = e < b.ne;
  if (active && sub < 10) {
    const int g = b.conn[sub * b.ne + e];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s_u[el][3 * sub + k] = u[3 * g + k];
      if (sub < 4) s_x[el][3 * sub + k] = X[3 * g + k];
    }
  }
  if (sub == 0) s_ok[el] = active;
  __syncthreads();
  double* sA = smem + (size_t)el * ASE;  // A and B take turns in the same memory
  double* sB = smem + (size_t)el * BSE;
  double acc[45];
#pragma unroll
  for (int k = 0; k < 45; ++k) acc[k] = 0.0;
  bool sound = true;  // no doubtful determinant at this thread's points
  for (int q0 = 0; q0 < b.nq; q0 += QT) {
    const int q = q0 + sub;
    if (q0 > 0) __syncthreads();  // the previous tile has been summed
    // ---- A ----
    if (threadIdx.x < QT * 16 / 2) {
      const int t = 2 * threadIdx.x;
      const int r = t / 16;
#pragma unroll
      for (int k = 0; k < 2; ++k) s_w[r][t % 16 + k] = q0 + r < b.nq ? weights[(size_t)(q0 + r) * 16 + t % 16 + k] : 0.0;
    }
    if (active && q < b.nq) {
      double J[9], Ji[9];
      tet4_jacobian(s_x[el], J);
      const double detJ = cofactors(J, Ji);  // Ji: cofactor matrix = det J * J^-T
      const double invJ = 1.0 / detJ;
      const double xi[3] = {b.qp[3 * q], b.qp[3 * q + 1], b.qp[3 * q + 2]};
      double p[4], h[4][3];
      tet4_psi(xi, p);
      // h_v = (4 l_v - 1) u_v + 4 sum over the edges (v, w) of l_w u_(v,w):
      // F = I + sum_v h_v g_v^T
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int c = 0; c < 3; ++c) h[v][c] = (4.0 * p[v] - 1.0) * s_u[el][3 * v + c];
#pragma unroll
      for (int n = 0; n < 6; ++n) {
        const int a = n == 0 || n == 2 || n == 3 ? 0 : (n == 1 || n == 5 ? 1 : 2);
        const int d = n == 0 ? 1 : (n == 1 || n == 2 ? 2 : 3);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double un = 4.0 * s_u[el][12 + 3 * n + c];
          h[a][c] += p[d] * un;
          h[d][c] += p[a] * un;
        }
      }
      double g[3][3];  // g_1, g_2, g_3
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        double gr[3];
        tet4_g(x + 1, gr);
#pragma unroll
        for (int k = 0; k < 3; ++k) g[x][k] = (Ji[3 * k] * gr[0] + Ji[3 * k + 1] * gr[1] + Ji[3 * k + 2] * gr[2]) * invJ;
      }
      double F[9];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k)
          F[3 * c + k] = (c == k ? 1.0 : 0.0) + (h[1][c] - h[0][c]) * g[0][k] + (h[2][c] - h[0][c]) * g[1][k] +
                         (h[3][c] - h[0][c]) * g[2][k];
      const double mu = b.emat ? b.emat[2 * e] : mat.mu, lam = b.emat ? b.emat[2 * e + 1] : mat.lambda;
      QpPair<double> qp;
      double M1[9];
      double scale = 0.0;
#pragma unroll
      for (int k = 0; k < 9; ++k) scale = fmax(scale, fabs(J[k]));
      sound &= point_state(mat.kind, F, mu, lam, qp, M1) && !det_doubtful(detJ, Ji, scale);
      const double sc = sqrt(b.qw[q] * fabs(detJ));
      double v[3][9];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
#pragma unroll
        for (int k = 0; k < 3; ++k) v[x][k] = g[x][k] * sc;
        mat3vec(F, v[x], v[x] + 3);
        mat3vec(M1, v[x], v[x] + 6);
      }
      double* o = sA + (size_t)sub * AS;
      // diagonal blocks 11, 22, 33 (upper entries), then 12, 13, 23
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        double k9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        pair_block(mat.kind, qp, v[x], v[x], k9);
        o[6 * x] = k9[0];
        o[6 * x + 1] = k9[1];
        o[6 * x + 2] = k9[2];
        o[6 * x + 3] = k9[4];
        o[6 * x + 4] = k9[5];
        o[6 * x + 5] = k9[8];
      }
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        double k9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        pair_block(mat.kind, qp, v[n < 2 ? 0 : 1], v[n == 0 ? 1 : 2], k9);
#pragma unroll
        for (int k = 0; k < 9; ++k) o[18 + 9 * n + k] = k9[k];
      }
    }
    __syncthreads();
    // ---- B ----
    const int nql = min(QT, b.nq - q0);
    if (sub < NW) {
#pragma unroll 1
      for (int r = 0; r < nql; ++r) {
        const double w = s_w[r][sub];
        const double2* a2 = reinterpret_cast<const double2*>(sA + (size_t)r * AS);
#pragma unroll
        for (int k = 0; k < 22; ++k) {
          const double2 t = a2[k];
          acc[2 * k] += w * t.x;
          acc[2 * k + 1] += w * t.y;
        }
        acc[44] += w * sA[(size_t)r * AS + 44];
      }
    }
  }
  __syncthreads();  // the points' blocks make room for the moments'
  if (sub < NW) {
    double* o = sB + sub * 90;
    // full blocks of x, y in 1 .. 3; off-diagonal ones as rows x < columns y
    auto at = [&](int x, int y, int i, int j) -> double {
      if (x == y) {
        const int lo = i < j ? i : j, hi = i < j ? j : i;
        return acc[6 * (x - 1) + (lo == 0 ? hi : (lo == 1 ? hi + 2 : 5))];
      }
      const int n = x + y - 3;  // 12, 13, 23
      return x < y ? acc[18 + 9 * n + 3 * i + j] : acc[18 + 9 * n + 3 * j + i];
    };
    double z[3][9];  // blocks 01, 02, 03
#pragma unroll
    for (int y = 1; y < 4; ++y)
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          z[y - 1][3 * i + j] = -(at(1, y, i, j) + at(2, y, i, j) + at(3, y, i, j));
          o[9 * sym4(0, y) + 3 * i + j] = z[y - 1][3 * i + j];
        }
#pragma unroll
    for (int k = 0; k < 9; ++k) o[k] = -(z[0][k] + z[1][k] + z[2][k]);
#pragma unroll
    for (int x = 1; x < 4; ++x)
#pragma unroll
      for (int y = x; y < 4; ++y)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) o[9 * sym4(x, y) + 3 * i + j] = at(x, y, i, j);
  }
  if (!sound)
    for (int q = sub; q < b.nq; q += TPE)
      if (tet10_singular(mat.kind, s_x[el], s_u[el], b.qp + 3 * (size_t)q)) s_ok[el] = 0;
  __syncthreads();
  // ---- C ---- (a thread decodes the terms of one pair's row once, for half of
  // the CTA's elements)
  const int e0 = blockIdx.x * EPC, nel = min(EPC, b.ne - e0);
  for (int t = threadIdx.x; t < 2 * NPAIR * 3; t += EPC * TPE) {
    const int half = t / (NPAIR * 3), r = t - half * (NPAIR * 3);
    const int p = r / 3, i = r - 3 * p;
    int at[4][2];  // offset of the row's first value and stride between its three
    double w[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int c = c_terms.at[p][n], k = (c >> 12) - 8;
      w[n] = (double)(k == 7 ? 16 : k);
      at[n][0] = (c & 2047) + (c & 2048 ? i : 3 * i);
      at[n][1] = c & 2048 ? 3 : 1;
    }
    for (int le = half * (EPC / 2); le < min(nel, (half + 1) * (EPC / 2)); ++le) {
      if (!s_ok[le]) continue;
      const double* B = smem + (size_t)le * BSE;
      double* o = pblk + ((size_t)(e0 + le) * NPAIR + p) * 9 + 3 * i;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double k = w[0] * B[at[0][0] + j * at[0][1]];
#pragma unroll
        for (int n = 1; n < 4; ++n) k += w[n] * B[at[n][0] + j * at[n][1]];
        o[j] = k;
      }
    }
  }
  if (active && sub == 0 && !s_ok[el]) set_error(err, HOEFEM_ERR_SINGULAR);
}

}  // namespace

bool stiffness_moments_eligible(const Block& blk) {
  return blk.kind == HOEFEM_ELEM_TET10 && blk.uniform && !blk.qw.empty();
}

// The block's node-pair blocks pblk[(e 55 + p) 9 + 3 i + j] (FP64).
void launch_stiffness_moments(const Model& m, const Block& blk, const MatDev& mat, const double* u, double* pblk,
                              cudaStream_t s) {
  if (!blk.d_moment_w.p) {
    std::vector<double> w(blk.qw.size() * 16, 0.0);
    for (size_t q = 0; q < blk.qw.size(); ++q) {
      const double* xi = blk.qp.data() + 3 * q;
      double p[4];
      p[0] = -0.5 * xi[0] - 0.5 * xi[1] - 0.5 * xi[2] - 0.5;
      for (int k = 0; k < 3; ++k) p[k + 1] = 0.5 * xi[k] + 0.5;
      for (int v = 0; v < 4; ++v) {
        for (int x = v; x < 4; ++x) w[16 * q + sym4(v, x)] = p[v] * p[x];
        w[16 * q + 10 + v] = p[v];
      }
      w[16 * q + 14] = 1.0;
    }
    blk.d_moment_w.upload(w, s);
    HOEFEM_CUDA(cudaStreamSynchronize(s));
  }
  const size_t smem = sizeof(double) * (size_t)EPC * (BSE > ASE ? BSE : ASE);
  HOEFEM_CUDA(cudaFuncSetAttribute(k_stiffness_moments, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  (note_launch(), k_stiffness_moments<<<(int)((blk.ne + EPC - 1) / EPC), EPC * TPE, smem, s>>>(
                      blk.dev(), m.d_X.p, u, blk.d_moment_w.p, mat, m.d_err.p, pblk));
  HOEFEM_CUDA(cudaGetLastError());
}

}  // namespace hoefem
