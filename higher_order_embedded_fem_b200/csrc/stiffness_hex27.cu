// FP64 element stiffness of Hex27 elements on the FP64 tensor cores.
//
// Reference: fenris/src/assembly.rs:746-797 (element stiffness), :252-314 +
// :1042-1075 (colored CSR scatter), fenris/src/solid/materials.rs:689-743
// (stress contraction).
//
// With gr_I(q) the reference gradient of node I and A_q(x, y) the 3 x 3 tangent
// contraction of the reference directions x, y (times w |det J|),
//   K_IJ[i][j] = sum_q sum_x gr_I[x] V^ij_J[q, x],  V^ij_J[q, x] = sum_y A_q(x, y)[i][j] gr_J[y].
// For each component pair (i, j) that is a product G^T V of node x 3Q by 3Q x node
// matrices with the same G; K^ji = (K^ij)^T leaves six pairs, and of the three with
// i = j one triangle.  Against the rank-structured pair loop (52 operations and 31
// shared-memory values per node pair and point, which bound it) 27 operations, and
// the operands of an 8 x 8 x 4 product come as one value a lane.  The products cover
// nodes 0 .. 23 in 8 x 8 tiles (9 and 6 of them); the columns of nodes 24 .. 26 of all
// nine pairs make one more product of 27 columns (16 tiles).  61 tiles instead of 78
// with 27 padded to 32.
//
// Persistent CTAs (two per SM) of two producer and four consumer warps, one of these
// per SM quadrant, over a ring of two stages.  An item is up to QA points of an
// element.
//  producer (the warp of the stage), lane = point: F, material state, the tangent
//     blocks A_q(x, y) (45 values) into the stage, then G (lane = node)
//  consumer 0 .. 2: a pair i < j and a pair i = j (15 tiles), consumer 3: the last
//     columns (16): per four points V (lane = column) into its own shared memory,
//     then three k-steps, accumulators in registers; after the element's last item
//     its 378 node-pair blocks in the stage's memory, from there to the staging
//     buffer, the dense element matrix or the CSR values
// The point phase is a chain of some 800 operations of a single warp: with one
// element per CTA and a barrier behind it the products waited for it (307 us).
// Stages are handed over by named barriers.  FP64 mma runs at the rate of the FP64
// pipe (36.9 TFLOP/s measured, against 32.2 of plain FMA loops): 11.7 k
// multiply-adds per point.  4,608 elements of 8 to 27 points: 458 -> 179 us (of
// which the products are a third; the rest is latency at two consumer warps per quadrant).
// Relative error against extended precision 2.8e-16 to 3.1e-16 (cylinders of 8^3 and
// 6^3 cells) where the pair loop had 4.9e-16 to 4.1e-16: the Jacobian comes from
// edges, not from absolute coordinates.
#include <cuda_runtime.h>

#include <algorithm>

#include "element_math.cuh"
#include "internal.h"

namespace hoefem {

namespace {

constexpr int NN = 27, NP = NN * (NN + 1) / 2;
constexpr int CW = 4;                // consumer warps
constexpr int STAGES = 2;            // a producer warp each
constexpr int TPB = 32 * (CW + STAGES);
constexpr int QA = 28;               // points of an item: every rule of up to 3 x 3 x 3 points is one
constexpr int QB = 4;                // points of a consumer's tile: three k-steps
constexpr int NT = 24;               // nodes of the full tiles
constexpr int RS = 36, VS = 28;      // rows of G, V: 4 or 12 mod 16 doubles, so a fragment's 4 rows x 8 columns miss each other's banks
constexpr int TS = 50;               // A_q: 16 per consumer (9, 6, pad), 2 pad
constexpr int DU = 90, DE = 36, DX = 24;
constexpr int D_PROD = DU + DE + DX + 18 * QA;      // a producer's element data
constexpr int D_STAGE = QA * TS + 3 * QA * RS;      // T, G; later the pair blocks
constexpr int D_V = 2 * 3 * QB * VS;                // a consumer's V
constexpr int DOUBLES = STAGES * (D_STAGE + D_PROD) + CW * D_V;
static_assert(3 * QB * RS <= D_V && QA <= 32 && QA % QB == 0 && NP * 9 <= D_STAGE && D_STAGE % 2 == 0 && D_PROD % 2 == 0, "layout");
constexpr size_t SMEM = sizeof(double) * (size_t)DOUBLES;
constexpr int BAR_FULL = 1, BAR_EMPTY = BAR_FULL + STAGES, BAR_CONSUMERS = BAR_EMPTY + STAGES;

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void mma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// A_q(x, y)[i][j] = A_q(y, x)[j][i] in the point's values: per consumer 0 .. 2 its
// pair i < j by (x, y), then its pair i = j by x <= y.
__device__ __forceinline__ constexpr int tangent_at(int x, int y, int i, int j) {
  if (i != j) return 16 * (i + j - 1) + (i < j ? 3 * x + y : 3 * y + x);
  const int lo = x < y ? x : y, hi = x < y ? y : x;
  return 16 * i + 9 + (lo == 0 ? hi : (lo == 1 ? hi + 2 : 5));
}

// Consumer W's products over nq points: pair i < j in tiles 0 .. 8 of acc, pair i = j
// in 9 .. 14 (lower triangle by rows).
template <int W>
__device__ __forceinline__ void contract(const double* T, const double* G, double* V, int nq, double (&acc)[16][2]) {
  const int lane = threadIdx.x & 31;
  const double* ga = G + (lane & 3) * RS + (lane >> 2);
  const double* vb = V + (lane & 3) * VS + (lane >> 2);
#pragma unroll 1
  for (int q0 = 0; q0 < nq; q0 += QB) {
    if (lane < NT) {
#pragma unroll
      for (int r = 0; r < QB; ++r) {
        const double2* t2 = reinterpret_cast<const double2*>(T + (q0 + r) * TS + 16 * W);
        const double* g = G + 3 * (q0 + r) * RS + lane;
        const double g0 = g[0], g1 = g[RS], g2 = g[2 * RS];
        double t[16];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const double2 v = t2[k];
          t[2 * k] = v.x;
          t[2 * k + 1] = v.y;
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          V[(3 * r + x) * VS + lane] = t[3 * x] * g0 + t[3 * x + 1] * g1 + t[3 * x + 2] * g2;
          V[(3 * (QB + r) + x) * VS + lane] = t[tangent_at(x, 0, 0, 0)] * g0 + t[tangent_at(x, 1, 0, 0)] * g1 +
                                              t[tangent_at(x, 2, 0, 0)] * g2;
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      double a[3], v[3], d[3];
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        a[n] = ga[(3 * q0 + 4 * s) * RS + 8 * n];
        v[n] = vb[4 * s * VS + 8 * n];
        d[n] = vb[(3 * QB + 4 * s) * VS + 8 * n];
      }
#pragma unroll
      for (int ti = 0; ti < 3; ++ti)
#pragma unroll
        for (int tj = 0; tj < 3; ++tj) {
          mma_8x8x4(acc[3 * ti + tj], a[ti], v[tj]);
          if (tj <= ti) mma_8x8x4(acc[9 + ti * (ti + 1) / 2 + tj], a[ti], d[tj]);
        }
    }
    __syncwarp();
  }
}

// The product of the last columns: column c is component pair c / 3 (of nine) of
// node NT + c % 3, rows are all nodes.
__device__ __forceinline__ void contract_last(const double* T, const double* G, double* V, int nq, double (&acc)[16][2]) {
  const int lane = threadIdx.x & 31;
  const double* ga = G + (lane & 3) * RS + (lane >> 2);
  const double* vb = V + (lane & 3) * RS + (lane >> 2);
  int at[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) at[k] = tangent_at(k / 3, k % 3, lane / 9, lane / 3 % 3);
#pragma unroll 1
  for (int q0 = 0; q0 < nq; q0 += QB) {
    if (lane < NN) {
#pragma unroll
      for (int r = 0; r < QB; ++r) {
        const double* t = T + (q0 + r) * TS;
        const double* g = G + 3 * (q0 + r) * RS + NT + lane % 3;
        const double g0 = g[0], g1 = g[RS], g2 = g[2 * RS];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          V[(3 * r + x) * RS + lane] = t[at[3 * x]] * g0 + t[at[3 * x + 1]] * g1 + t[at[3 * x + 2]] * g2;
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      double a[4], v[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        a[n] = ga[(3 * q0 + 4 * s) * RS + 8 * n];
        v[n] = vb[4 * s * RS + 8 * n];
      }
#pragma unroll
      for (int ti = 0; ti < 4; ++ti)
#pragma unroll
        for (int tj = 0; tj < 4; ++tj) mma_8x8x4(acc[4 * ti + tj], a[ti], v[tj]);
    }
    __syncwarp();
  }
}

// Place of node pair lo <= hi among the element's blocks (row node hi, column node lo).
__device__ __forceinline__ int pair_at(int lo, int hi) { return lo * NN - lo * (lo - 1) / 2 + hi - lo; }

// The tangent blocks and G of the points t0 .. t0 + nt of element e; true if none
// of the warp's points is singular.
__device__ __forceinline__ bool produce(const BlockDev& b, const MatDev& mat, int e, int q0, int nt, double* su,
                                        double* sT, double* sG) {
  double* se = su + DU;
  double* sx = se + DE;
  double* sp = sx + DX;
  const int lane = threadIdx.x & 31;
  const int nb = (nt + QB - 1) / QB * QB;
  bool sound = true;
  if (lane < nt) {
    const double* xq = b.qp + 3 * (size_t)(q0 + lane);
    const double xi[3] = {xq[0], xq[1], xq[2]};
    const double w = b.qw[q0 + lane];
    const double mu = b.emat ? b.emat[2 * e] : mat.mu, lam = b.emat ? b.emat[2 * e + 1] : mat.lambda;
    double H[9], J[9], C[9], F[9];
    {
      double p[9], d[9];
      hex27_axes(xi, p, d);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        sp[18 * lane + k] = p[k];
        sp[18 * lane + 9 + k] = d[k];
      }
      hex27_gradient(su, p, d, H);
    }
    hex8_jacobian_edges(se, xi, J);
    const double det = cofactors(J, C);  // J^-1[m][k] = C[3 k + m] / det
    const double inv = 1.0 / det;
    double scale = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) scale = fmax(scale, fabs(J[k]));
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k)
        F[3 * c + k] = (c == k ? 1.0 : 0.0) +
                       (H[3 * c] * C[3 * k] + H[3 * c + 1] * C[3 * k + 1] + H[3 * c + 2] * C[3 * k + 2]) * inv;
    QpPair<double> qp;
    double M1[9], v[3][9];
    sound = point_state(mat.kind, F, mu, lam, qp, M1) && !det_doubtful(det, C, scale);
    const double sc = sqrt(w * fabs(det)) * inv;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
#pragma unroll
      for (int k = 0; k < 3; ++k) v[x][k] = C[3 * k + x] * sc;
      mat3vec(F, v[x], v[x] + 3);
      mat3vec(M1, v[x], v[x] + 6);
    }
    double* t = sT + TS * lane;
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const int x = n < 3 ? n : (n == 5 ? 1 : 0), y = n < 3 ? n : (n == 3 ? 1 : 2);
      double k9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      pair_block(mat.kind, qp, v[x], v[y], k9);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (x < y || i <= j) t[tangent_at(x, y, i, j)] = k9[3 * i + j];
    }
  } else if (lane < nb) {  // a point that fills up the last tile
#pragma unroll
    for (int k = 0; k < 48; ++k) sT[TS * lane + k] = 0.0;
  }
  bool ok = true;
  if (!sound) ok = !hex27_singular(mat.kind, sx, su, b.qp + 3 * (size_t)(q0 + lane));
  __syncwarp();
  // G
  if (lane < NN) {
    const signed char* al = c_hex27_alpha[lane];
    const int i = al[0] + 1, j = al[1] + 1, k = al[2] + 1;
#pragma unroll 4
    for (int r = 0; r < nb; ++r) {
      const double* p = sp + 18 * min(r, nt - 1);
      const double px = p[i], py = p[3 + j], pz = p[6 + k];
      double* g = sG + 3 * r * RS + lane;  // (any finite value where T is zero)
      g[0] = p[9 + i] * py * pz;
      g[RS] = px * p[12 + j] * pz;
      g[2 * RS] = px * py * p[15 + k];
    }
  }
  return __all_sync(0xffffffffu, ok);
}

// The CTA's items in order: fn(element, first point, points, last item of the element).
template <class F>
__device__ __forceinline__ void for_each_item(const BlockDev& b, const int* __restrict__ elems, int count, F&& fn) {
  for (int n = blockIdx.x; n < count; n += gridDim.x) {
    const int e = elems ? elems[n] : n;
    if (b.scene_active && !b.scene_active[b.escene[e]]) continue;
    int q0, nq;
    quad_rule(b, e, q0, nq);
    int t0 = 0;
    do {
      fn(e, q0 + t0, min(QA, nq - t0), t0 == 0, t0 + QA >= nq);
      t0 += QA;
    } while (t0 < nq);
  }
}

__global__ void __launch_bounds__(TPB, 2) k_stiffness_hex27(const BlockDev b, const int* __restrict__ elems, int count,
                                                            const double* __restrict__ X, const double* __restrict__ u,
                                                            const int* __restrict__ adj_off,
                                                            const long long* __restrict__ base,
                                                            double* __restrict__ vals, MatDev mat, int* err,
                                                            double* __restrict__ stage, double* __restrict__ pblk) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_ok[STAGES];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int item = 0;
  if (warp >= CW) {
    // ---- producers ----
    const int st = warp - CW;
    double* sT = smem + st * D_STAGE;
    double* su = smem + STAGES * D_STAGE + CW * D_V + st * D_PROD;
    for_each_item(b, elems, count, [&](int e, int q0, int nt, bool, bool) {
      if (item++ % STAGES != st) return;
      if (lane < NN) {
        const int I = hex27_at(lane), g = b.conn[I * b.ne + e];
#pragma unroll
        for (int k = 0; k < 3; ++k) su[10 * (lane / 3) + 3 * (lane % 3) + k] = u[3 * g + k];
        if (I < 8) {
          const int corner = (lane % 3 >> 1) | (lane / 3 % 3 & 2) | (lane / 9 & 2) << 1;
#pragma unroll
          for (int k = 0; k < 3; ++k) su[DU + DE + 3 * corner + k] = X[3 * g + k];
        }
      }
      __syncwarp();
      for (int t = lane; t < DE; t += 32) su[DU + t] = hex8_edge(su + DU + DE, t);
      __syncwarp();
      if (item > STAGES) bar_sync(BAR_EMPTY + st, 32 * (CW + 1));
      const bool ok = produce(b, mat, e, q0, nt, su, sT, sT + QA * TS);
      if (lane == 0) s_ok[st] = ok;
      __syncwarp();
      bar_arrive(BAR_FULL + st, 32 * (CW + 1));
    });
    // the hand-backs of the last items
    for (int n = max(0, item - STAGES); n < item; ++n)
      if (n % STAGES == st) bar_sync(BAR_EMPTY + st, 32 * (CW + 1));
    return;
  }
  // ---- consumers: pairs 01 and 00, 02 and 11, 12 and 22, the last columns ----
  double* sV = smem + STAGES * D_STAGE + warp * D_V;
  double acc[16][2];
  bool ok = true;
  for_each_item(b, elems, count, [&](int e, int, int nt, bool first, bool last) {
    const int st = item++ % STAGES;
    double* sT = smem + st * D_STAGE;
    const double* sG = sT + QA * TS;
    if (first) {
      ok = true;
#pragma unroll
      for (int n = 0; n < 16; ++n) acc[n][0] = acc[n][1] = 0.0;
    }
    bar_sync(BAR_FULL + st, 32 * (CW + 1));
    ok &= s_ok[st] != 0;
    switch (warp) {
      case 0: contract<0>(sT, sG, sV, nt, acc); break;
      case 1: contract<1>(sT, sG, sV, nt, acc); break;
      case 2: contract<2>(sT, sG, sV, nt, acc); break;
      default: contract_last(sT, sG, sV, nt, acc); break;
    }
    if (last && ok) {
      double* sK = sT;  // every warp has read the stage
      bar_sync(BAR_CONSUMERS, 32 * CW);
      const int row = lane >> 2, col = 2 * (lane & 3);
      if (warp < 3) {
        const int ci = warp == 2 ? 1 : 0, cj = warp == 0 ? 1 : 2;
#pragma unroll
        for (int ti = 0; ti < 3; ++ti)
#pragma unroll
          for (int tj = 0; tj < 3; ++tj)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int I = 8 * ti + row, Jn = 8 * tj + col + r;
              const double v = acc[3 * ti + tj][r];
              if (I >= Jn) sK[pair_at(Jn, I) * 9 + 3 * ci + cj] = v;
              if (I <= Jn) sK[pair_at(I, Jn) * 9 + 3 * cj + ci] = v;
              if (tj <= ti && I >= Jn) sK[pair_at(Jn, I) * 9 + 4 * warp] = acc[9 + ti * (ti + 1) / 2 + (tj <= ti ? tj : 0)][r];
            }
      } else {
#pragma unroll
        for (int n = 0; n < 16; ++n)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int I = 8 * (n / 4) + row, c = 8 * (n % 4) + col + r, Jn = NT + c % 3, i = c / 9, j = c / 3 % 3;
            if (I >= NN || c >= NN) continue;
            if (I < NT) sK[pair_at(I, Jn) * 9 + 3 * j + i] = acc[n][r];
            else if (I >= Jn) sK[pair_at(Jn, I) * 9 + 3 * i + j] = acc[n][r];
          }
      }
      bar_sync(BAR_CONSUMERS, 32 * CW);
      if (pblk) {
        // node-pair blocks, pblk[(e NP + p) 9 + 3 i + j], for the gather into the CSR values
        double2* o = reinterpret_cast<double2*>(pblk + (size_t)e * (NP * 9));
        const double2* k2 = reinterpret_cast<const double2*>(sK);
        for (int t = threadIdx.x; t < NP * 9 / 2; t += 32 * CW) o[t] = k2[t];
      } else {
        const int* em = b.emap + (size_t)e * NN * NN;
        for (int t = threadIdx.x; t < NN * NN; t += 32 * CW) {
          const int I = t / NN, Jn = t - NN * I;
          const bool tr = I < Jn;
          const int hi = tr ? Jn : I, lo = tr ? I : Jn;
          const double* k9 = sK + (lo * NN - lo * (lo - 1) / 2 + hi - lo) * 9;
          double* o;
          int ld;
          if (stage) {  // dense element matrix, row-major 81 x 81
            ld = 3 * NN;
            o = stage + (size_t)e * ld * ld + 3 * I * ld + 3 * Jn;
          } else {
            const int g = b.conn[I * b.ne + e];
            ld = 3 * (adj_off[g + 1] - adj_off[g]);
            o = vals + base[g] + em[t];
          }
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const double v = tr ? k9[3 * j + i] : k9[3 * i + j];
              o[i * ld + j] = stage ? v : o[i * ld + j] + v;
            }
        }
      }
    } else if (last && threadIdx.x == 0) {
      set_error(err, HOEFEM_ERR_SINGULAR);
    }
    bar_arrive(BAR_EMPTY + st, 32 * (CW + 1));
  });
}

}  // namespace

// count elements (elems, or all by number) into pblk, stage or vals.
void launch_stiffness_hex27(const Model& m, const Block& blk, const int* elems, int count, const MatDev& mat,
                            const double* u, double* vals, double* stage, double* pblk, cudaStream_t s) {
  HOEFEM_CUDA(cudaFuncSetAttribute(k_stiffness_hex27, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
  const int grid = std::min(count, 2 * device_sms());
  (note_launch(), k_stiffness_hex27<<<grid, TPB, SMEM, s>>>(blk.dev(), elems, count, m.d_X.p, u, m.d_adj_off.p,
                                                            m.d_base.p, vals, mat, m.d_err.p, stage, pblk));
  HOEFEM_CUDA(cudaGetLastError());
}

}  // namespace hoefem
