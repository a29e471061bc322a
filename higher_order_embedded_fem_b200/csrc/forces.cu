// Internal forces f_e(:, I) -= P J^-T grad N_I w |det J| of Tet10 and Hex27
// elements (FP64), for any quadrature rule (one per block or per element).
//
// Reference: fenris/src/assembly.rs:673-711 (element force), :915-966 (colored
// scatter), fenris/src/solid/materials.rs:177-346 (stress).
//
// A lane owns a quadrature point: the displacement gradient, the stress and
// Q = -w |det J| P J^-T of its point, without a reduction over lanes.  The node
// sums over the points follow from Q in shared memory, lanes owning sums.  (One
// lane per node instead takes nine FP64 warp sums of five shuffles per point and
// repeats the Jacobian and the stress on all 32 lanes: that bound the Hex27
// kernel.)  Whole-block launches go by element number, so that neighbouring warps
// read neighbouring connectivity; colored launches take the color's list.
#include <cuda_runtime.h>

#include "element_math.cuh"
#include "internal.h"

namespace hoefem {

namespace {

constexpr int TPB = 128;

// First Piola-Kirchhoff stress of F; false where F is doubtful (det_doubtful).
__device__ __forceinline__ bool point_stress(int kind, const double* F, double mu0, double lam0, double* P) {
  if (kind == HOEFEM_MAT_SNH) {
    const double mu = 4.0 / 3.0 * mu0, lam = lam0 + (1.0 - 2.0 / 12.0) * mu0;
    const double alpha = 1.0 + mu / lam * 0.75;
    double IC = 0.0, C[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) IC += F[k] * F[k];
    const double J = cofactors(F, C);
    const double cf = mu * (1.0 - 1.0 / (IC + 1.0)), cj = lam * (J - alpha);
#pragma unroll
    for (int k = 0; k < 9; ++k) P[k] = F[k] * cf + C[k] * cj;
    return !det_doubtful(J, C, 1.0);
  }
  QpState<double> st;
  stvk_state(F, mu0, lam0, st, true);
#pragma unroll
  for (int k = 0; k < 9; ++k) P[k] = st.P[k];
  return true;
}

// Q[3 i + m] = -w |det J| sum_k P[i][k] (J^-1)[m][k] from the displacement's
// reference gradient H and the Jacobian, so that node I gets sum_m Q[i][m] dN_I/dxi_m;
// false where J or F is doubtful.
__device__ __forceinline__ bool point_flux(int kind, const double* H, const double* J, double w, double mu, double lam,
                                           double* Q) {
  double C[9];
  const double det = cofactors(J, C);  // J^-1[m][k] = C[3 k + m] / det
  const double inv = 1.0 / det;
  double scale = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) scale = fmax(scale, fabs(J[k]));
  const bool firm = !det_doubtful(det, C, scale);
  double F[9];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k)
      F[3 * c + k] = (c == k ? 1.0 : 0.0) + (H[3 * c] * C[3 * k] + H[3 * c + 1] * C[3 * k + 1] + H[3 * c + 2] * C[3 * k + 2]) * inv;
  double P[9];
  const bool sound = point_stress(kind, F, mu, lam, P) && firm;
  const double sc = det > 0.0 ? -w : w;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int m = 0; m < 3; ++m)
      Q[3 * i + m] = sc * (P[3 * i] * C[m] + P[3 * i + 1] * C[3 + m] + P[3 * i + 2] * C[6 + m]);
  return sound;
}

// ============================================================================
// Tet10: 16 lanes per element, two elements per warp, tiles of 16 points.  With
// l_v the barycentric functions, the gradient of the displacement is linear in
// them: H = sum_v l_v H_v with H_v its value at vertex v (4 u_(x,v) - u_x along
// an edge (x, v), 3 u_v at the vertex itself); and every node force is a
// combination of the twelve vectors M_v = sum_q l_v Q_q.  36 operations a point
// for each direction instead of 10 nodes x (gradient + 9) twice.  201,600 elements
// of 14 points: 721 -> 222 us (shared memory at 63 % of its peak, FP64 at 29 %; the rest
// is the latency of a point's chain at 16 warps per SM).
// ============================================================================
constexpr int T10_LANES = 16;
constexpr int T10_EPC = TPB / T10_LANES;
constexpr int T10_PS = 13;                                 // doubles per point: Q, l
constexpr int T10_ES = 30 + 12 + 36 + 16 * T10_PS + 1;     // per element, odd: the warp's two elements on different banks

__device__ __forceinline__ int tet10_edge_node(int a, int b) {  // a != b; 01 12 02 03 23 13
  const int lo = min(a, b), hi = max(a, b);
  return lo == 0 ? (hi == 1 ? 4 : hi + 4) : (lo == 2 ? 8 : (hi == 2 ? 5 : 9));
}

__global__ void __launch_bounds__(TPB) k_forces_tet10(const BlockDev b, const int* __restrict__ elems, int count,
                                                      const double* __restrict__ X, const double* __restrict__ u,
                                                      double* __restrict__ f, MatDev mat, int* err,
                                                      double* __restrict__ fst) {
  __shared__ double smem[T10_EPC * T10_ES];
  const int el = threadIdx.x / T10_LANES, sub = threadIdx.x % T10_LANES;
  const int idx = blockIdx.x * T10_EPC + el;
  const int e = idx < count ? (elems ? elems[idx] : idx) : 0;
  const bool active = idx < count && (!b.scene_active || b.scene_active[b.escene[e]]);
  double* su = smem + el * T10_ES;
  double* sx = su + 30;
  double* sh = sx + 12;   // H_v[v * 9 + 3 c + m], later M_v in the same order
  double* sp = sh + 36;
  int g = 0, q0 = 0, nq = 0;
  if (active) quad_rule(b, e, q0, nq);
  if (active && sub < 10) {
    g = b.conn[sub * b.ne + e];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      su[3 * sub + k] = u[3 * g + k];
      if (sub < 4) sx[3 * sub + k] = X[3 * g + k];
    }
  }
  __syncwarp();
  if (active) {
    for (int t = sub; t < 36; t += T10_LANES) {
      const int v = t / 9, c = (t - 9 * v) / 3, x = t % 3 + 1;
      const double dx = x == v ? 3.0 * su[3 * v + c] : 4.0 * su[3 * tet10_edge_node(x, v) + c] - su[3 * x + c];
      const double d0 = v == 0 ? 3.0 * su[c] : 4.0 * su[3 * tet10_edge_node(0, v) + c] - su[c];
      sh[t] = 0.5 * (dx - d0);
    }
  }
  __syncwarp();
  const double mu = b.emat ? b.emat[2 * e] : mat.mu, lam = b.emat ? b.emat[2 * e + 1] : mat.lambda;
  double J[9];
  bool sound = true;
  double acc[3] = {0.0, 0.0, 0.0};
  const int tiles = (max(nq, __shfl_xor_sync(0xffffffffu, nq, T10_LANES)) + T10_LANES - 1) / T10_LANES;
  if (active) tet4_jacobian(sx, J);
  for (int tile = 0; tile < tiles; ++tile) {
    const int q = tile * T10_LANES + sub;
    if (tile > 0) __syncwarp();  // the previous tile has been summed
    if (q < nq) {
      const double* xi = b.qp + 3 * (size_t)(q0 + q);
      const double x3[3] = {xi[0], xi[1], xi[2]};
      double l[4], H[9], Q[9];
      tet4_psi(x3, l);
#pragma unroll
      for (int k = 0; k < 9; ++k) H[k] = l[0] * sh[k] + l[1] * sh[9 + k] + l[2] * sh[18 + k] + l[3] * sh[27 + k];
      sound &= point_flux(mat.kind, H, J, b.qw[q0 + q], mu, lam, Q);
      double* o = sp + sub * T10_PS;
#pragma unroll
      for (int k = 0; k < 9; ++k) o[k] = Q[k];
#pragma unroll
      for (int v = 0; v < 4; ++v) o[9 + v] = l[v];
    }
    __syncwarp();
    if (sub < 12) {  // M_v[c][m] of v = sub / 3, m = sub % 3
      const int nql = min(T10_LANES, nq - tile * T10_LANES);
      const double* o = sp + sub % 3;
      const double* l = sp + 9 + sub / 3;
      for (int r = 0; r < nql; ++r, o += T10_PS, l += T10_PS) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += *l * o[3 * c];
      }
    }
  }
  bool ok = true;
  if (!sound)
    for (int q = sub; q < nq; q += T10_LANES) ok &= !tet10_singular(mat.kind, sx, su, b.qp + 3 * (size_t)(q0 + q));
  ok = ((__ballot_sync(0xffffffffu, ok) >> (threadIdx.x & 16)) & 0xffffu) == 0xffffu;
  if (sub < 12) {
#pragma unroll
    for (int c = 0; c < 3; ++c) sh[9 * (sub / 3) + 3 * c + sub % 3] = acc[c];
  }
  __syncwarp();
  if (!active) return;
  if (!ok) {
    if (sub == 0) set_error(err, HOEFEM_ERR_SINGULAR);
    return;
  }
  // the derivative along l_x: x = 1 .. 3 take half of a reference direction each,
  // x = 0 minus their sum
  auto along = [&](int x, int v, int c) {
    const double* r = sh + 9 * v + 3 * c;
    return x == 0 ? -0.5 * (r[0] + r[1] + r[2]) : 0.5 * r[x - 1];
  };
  for (int t = sub; t < 30; t += T10_LANES) {
    const int I = t / 3, c = t - 3 * I;
    double v;
    if (I < 4) {
      v = 4.0 * along(I, I, c) - (along(I, 0, c) + along(I, 1, c) + along(I, 2, c) + along(I, 3, c));
    } else {
      const int a = c_tet10_edge[I - 4][0], d = c_tet10_edge[I - 4][1];
      v = 4.0 * (along(a, d, c) + along(d, a, c));
    }
    if (fst) fst[(size_t)e * 30 + t] = v;
    else f[3 * b.conn[I * b.ne + e] + c] += v;
  }
}

// ============================================================================
// Hex27: a warp per element, tiles of 32 points.  The lane of a point sums the
// displacement gradient axis by axis (270 operations; 27 nodes x 3 x 3 directly
// plus the gradients' products), the lane of a node then adds the points'
// contributions in point order from Q and the one-dimensional functions.
// 4,608 elements of 8 to 27 points: 168 -> 29 us, bound by the latency of one
// element (all of them are resident at once).
// ============================================================================
constexpr int H27_PS = 30;                         // doubles per point: Q (9), phi (9), phi' (9); 16-byte rows
constexpr int H27_U = 90, H27_X = 24, H27_E = 36;  // node displacements (rows of 10), corners, edges
constexpr int H27_WS = H27_U + H27_E + H27_X + 32 * H27_PS;

__global__ void __launch_bounds__(TPB, 4) k_forces_hex27(const BlockDev b, const int* __restrict__ elems, int count,
                                                      const double* __restrict__ X, const double* __restrict__ u,
                                                      double* __restrict__ f, MatDev mat, int* err,
                                                      double* __restrict__ fst) {
  __shared__ __align__(16) double smem[(TPB / 32) * H27_WS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int idx = blockIdx.x * (TPB / 32) + warp;
  if (idx >= count) return;
  const int e = elems ? elems[idx] : idx;
  if (b.scene_active && !b.scene_active[b.escene[e]]) return;
  double* su = smem + warp * H27_WS;
  double* se = su + H27_U;
  double* sx = se + H27_E;
  double* sp = sx + H27_X;
  int q0, nq;
  quad_rule(b, e, q0, nq);
  const double mu = b.emat ? b.emat[2 * e] : mat.mu, lam = b.emat ? b.emat[2 * e + 1] : mat.lambda;
  const int I = lane < 27 ? hex27_at(lane) : 0;  // lane in axis order -> node
  int g = 0;
  if (lane < 27) {
    g = b.conn[I * b.ne + e];
#pragma unroll
    for (int k = 0; k < 3; ++k) su[lane + lane / 3 * 7 + (lane % 3) * 2 + k] = u[3 * g + k];
    if (I < 8) {
      const int corner = (lane % 3 >> 1) | (lane / 3 % 3 & 2) | (lane / 9 & 2) << 1;
#pragma unroll
      for (int k = 0; k < 3; ++k) sx[3 * corner + k] = X[3 * g + k];
    }
  }
  __syncwarp();
  for (int t = lane; t < H27_E; t += 32) se[t] = hex8_edge(sx, t);
  __syncwarp();
  const int i = lane % 3, j = lane / 3 % 3, k = lane / 9;
  double acc[3] = {0.0, 0.0, 0.0};
  bool sound = true;
  for (int t0 = 0; t0 < nq; t0 += 32) {
    if (t0 > 0) __syncwarp();  // the previous tile has been summed
    if (t0 + lane < nq) {
      const double* xq = b.qp + 3 * (size_t)(q0 + t0 + lane);
      const double xi[3] = {xq[0], xq[1], xq[2]};
      double p[9], d[9], H[9], J[9], Q[9];
      hex27_axes(xi, p, d);
      hex27_gradient(su, p, d, H);
      hex8_jacobian_edges(se, xi, J);
      sound &= point_flux(mat.kind, H, J, b.qw[q0 + t0 + lane], mu, lam, Q);
      double2* o = reinterpret_cast<double2*>(sp + lane * H27_PS);
      o[0] = make_double2(Q[0], Q[1]);
      o[1] = make_double2(Q[2], Q[3]);
      o[2] = make_double2(Q[4], Q[5]);
      o[3] = make_double2(Q[6], Q[7]);
      o[4] = make_double2(Q[8], p[0]);
#pragma unroll
      for (int r = 0; r < 4; ++r) o[5 + r] = make_double2(p[2 * r + 1], p[2 * r + 2]);
#pragma unroll
      for (int r = 0; r < 4; ++r) o[9 + r] = make_double2(d[2 * r], d[2 * r + 1]);
      sp[lane * H27_PS + 26] = d[8];
    }
    __syncwarp();
    const int nql = min(32, nq - t0);
    if (lane < 27) {
#pragma unroll 2
      for (int r = 0; r < nql; ++r) {
        const double* o = sp + r * H27_PS;
        const double2* o2 = reinterpret_cast<const double2*>(o);
        const double2 a0 = o2[0], a1 = o2[1], a2 = o2[2], a3 = o2[3];
        const double q8 = o[8];
        const double px = o[9 + i], py = o[12 + j], pz = o[15 + k];
        const double gx = o[18 + i] * py * pz, gy = px * o[21 + j] * pz, gz = px * py * o[24 + k];
        acc[0] += a0.x * gx + a0.y * gy + a1.x * gz;
        acc[1] += a1.y * gx + a2.x * gy + a2.y * gz;
        acc[2] += a3.x * gx + a3.y * gy + q8 * gz;
      }
    }
  }
  bool ok = true;
  if (!sound)
    for (int q = lane; q < nq; q += 32) ok &= !hex27_singular(mat.kind, sx, su, b.qp + 3 * (size_t)(q0 + q));
  if (!__all_sync(0xffffffffu, ok)) {
    if (lane == 0) set_error(err, HOEFEM_ERR_SINGULAR);
    return;
  }
  if (lane < 27) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (fst) fst[((size_t)e * 27 + I) * 3 + c] = acc[c];
      else f[3 * g + c] += acc[c];
    }
  }
}

}  // namespace

void launch_forces(const Model& m, const MatDev& mat, const double* u, double* f, cudaStream_t s) {
  for (const Block* bp : m.blocks) {
    BlockDev bd = bp->dev();
    auto launch = [&](const int* elems, int cnt, double* fst) {
      if (bp->kind == HOEFEM_ELEM_TET10)
        (note_launch(), k_forces_tet10<<<(cnt + T10_EPC - 1) / T10_EPC, TPB, 0, s>>>(bd, elems, cnt, m.d_X.p, u, f, mat,
                                                                                      m.d_err.p, fst));
      else
        (note_launch(), k_forces_hex27<<<(cnt + TPB / 32 - 1) / (TPB / 32), TPB, 0, s>>>(bd, elems, cnt, m.d_X.p, u, f,
                                                                                          mat, m.d_err.p, fst));
    };
    if (stiffness_pairs_eligible(m, *bp)) {
      // every element in one launch into per-element node forces, then the
      // per-node gather (element order)
      double* fst = forces_stage_buffer(m, *bp, s);
      if (bp->ne > 0) launch(nullptr, (int)bp->ne, fst);
      HOEFEM_CUDA(cudaGetLastError());
      forces_gather(m, *bp, f, s);
    } else {
      for_each_color(*bp, [&](const int* elems, int cnt) { launch(elems, cnt, nullptr); });
    }
  }
  HOEFEM_CUDA(cudaGetLastError());
}

}  // namespace hoefem
