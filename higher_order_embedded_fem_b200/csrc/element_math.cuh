// Device math shared by the element kernels: reference Tet10 / Hex27 shape
// function gradients, the Hex8 / Tet4 geometry Jacobians, the materials
// (stable Neo-Hookean, St. Venant-Kirchhoff) and the node-pair stiffness
// block of one quadrature point.
//
// Reference: fenris/src/element.rs (Tet10 1921-1947, Hex27 basis),
// fenris/src/solid/materials.rs (stress and its contraction 689-743).
#pragma once

#include <cuda_runtime.h>

#include "internal.h"

namespace hoefem {
namespace {

__constant__ signed char c_hex27_alpha[27][3] = {
    {-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1}, {-1, -1, 1}, {1, -1, 1}, {1, 1, 1}, {-1, 1, 1},
    {0, -1, -1},  {-1, 0, -1}, {-1, -1, 0}, {1, 0, -1}, {1, -1, 0}, {0, 1, -1}, {1, 1, 0}, {-1, 1, 0},
    {0, -1, 1},   {-1, 0, 1},  {1, 0, 1},   {0, 1, 1},  {0, 0, -1}, {0, -1, 0}, {-1, 0, 0}, {1, 0, 0},
    {0, 1, 0},    {0, 0, 1},   {0, 0, 0}};
__constant__ signed char c_tet10_edge[6][2] = {{0, 1}, {1, 2}, {0, 2}, {0, 3}, {2, 3}, {1, 3}};

template <class R>
__device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void set_error(int* err, int code) { atomicCAS(err, 0, code); }

// ---- reference elements ----------------------------------------------------
template <class R>
__device__ __forceinline__ void tet4_psi(const R* xi, R* p) {
  p[0] = -R(0.5) * xi[0] - R(0.5) * xi[1] - R(0.5) * xi[2] - R(0.5);
  p[1] = R(0.5) * xi[0] + R(0.5);
  p[2] = R(0.5) * xi[1] + R(0.5);
  p[3] = R(0.5) * xi[2] + R(0.5);
}
// gradient of Tet4 basis function I (constant): column I of [[-.5,.5,0,0],[-.5,0,.5,0],[-.5,0,0,.5]]
template <class R>
__device__ __forceinline__ void tet4_g(int I, R* g) {
  g[0] = (I == 0) ? -R(0.5) : (I == 1 ? R(0.5) : R(0.0));
  g[1] = (I == 0) ? -R(0.5) : (I == 2 ? R(0.5) : R(0.0));
  g[2] = (I == 0) ? -R(0.5) : (I == 3 ? R(0.5) : R(0.0));
}
// Tet10 reference gradient of node I (element.rs:1921-1947)
template <class R>
__device__ __forceinline__ void tet10_grad(int I, const R* xi, R* g) {
  R p[4];
  tet4_psi(xi, p);
  if (I < 4) {
    R gi[3];
    tet4_g(I, gi);
    R f = R(4.0) * p[I] - R(1.0);
    g[0] = gi[0] * f; g[1] = gi[1] * f; g[2] = gi[2] * f;
  } else {
    int a = c_tet10_edge[I - 4][0], b = c_tet10_edge[I - 4][1];
    R ga[3], gb[3];
    tet4_g(a, ga);
    tet4_g(b, gb);
    R fb = R(4.0) * p[b], fa = R(4.0) * p[a];
    g[0] = ga[0] * fb + gb[0] * fa;
    g[1] = ga[1] * fb + gb[1] * fa;
    g[2] = ga[2] * fb + gb[2] * fa;
  }
}
template <class R>
__device__ __forceinline__ R tet10_phi(int I, const R* xi) {
  R p[4];
  tet4_psi(xi, p);
  if (I < 4) return p[I] * (R(2.0) * p[I] - R(1.0));
  return R(4.0) * p[c_tet10_edge[I - 4][0]] * p[c_tet10_edge[I - 4][1]];
}
template <class R>
__device__ __forceinline__ R phi_q(R a, R x) {
  R a2 = a * a, x2 = x * x;
  return (R(3.0) / R(2.0) * a2 - R(1.0)) * x2 + R(0.5) * a * x + R(1.0) - a2;
}
template <class R>
__device__ __forceinline__ R dphi_q(R a, R x) {
  R a2 = a * a;
  return R(2.0) * (R(3.0) / R(2.0) * a2 - R(1.0)) * x + R(0.5) * a;
}
template <class R>
__device__ __forceinline__ void hex27_grad(int I, const R* xi, R* g) {
  R a0 = c_hex27_alpha[I][0], a1 = c_hex27_alpha[I][1], a2 = c_hex27_alpha[I][2];
  R p0 = phi_q(a0, xi[0]), p1 = phi_q(a1, xi[1]), p2 = phi_q(a2, xi[2]);
  g[0] = dphi_q(a0, xi[0]) * p1 * p2;
  g[1] = p0 * dphi_q(a1, xi[1]) * p2;
  g[2] = p0 * p1 * dphi_q(a2, xi[2]);
}
template <class R>
__device__ __forceinline__ R hex27_phi(int I, const R* xi) {
  return phi_q((R)c_hex27_alpha[I][0], xi[0]) * phi_q((R)c_hex27_alpha[I][1], xi[1]) *
         phi_q((R)c_hex27_alpha[I][2], xi[2]);
}
// Jacobian of the trilinear Hex8 geometry from the 8 corners (smem, xyz per corner).
template <class R>
__device__ __forceinline__ void hex8_jacobian(const R* Xc, const R* xi, R* J) {
#pragma unroll
  for (int k = 0; k < 9; ++k) J[k] = R(0.0);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    R a0 = c_hex27_alpha[c][0], a1 = c_hex27_alpha[c][1], a2 = c_hex27_alpha[c][2];
    R l0 = (R(1.0) + a0 * xi[0]) / R(2.0), l1 = (R(1.0) + a1 * xi[1]) / R(2.0), l2 = (R(1.0) + a2 * xi[2]) / R(2.0);
    R g0 = a0 / R(2.0) * l1 * l2, g1 = l0 * a1 / R(2.0) * l2, g2 = l0 * l1 * a2 / R(2.0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      R x = Xc[3 * c + i];
      J[3 * i + 0] += x * g0;
      J[3 * i + 1] += x * g1;
      J[3 * i + 2] += x * g2;
    }
  }
}
// Jacobian of the affine Tet4 geometry: J(:,j) = R(0.5) (X_{j+1} - X_0)
template <class R>
__device__ __forceinline__ void tet4_jacobian(const R* Xc, R* J) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) J[3 * i + j] = -R(0.5) * Xc[i] + R(0.5) * Xc[3 * (j + 1) + i];
}

// ---- Hex27 in axis order -----------------------------------------------------
// Node of place i + 3 j + 9 k, coordinate -1, 0, 1 for i, j, k = 0, 1, 2.
__device__ const unsigned char g_hex27_at[27] = {0, 8,  1, 9, 20, 11, 3, 13, 2, 10, 21, 12, 22, 26,
                                                 23, 15, 24, 14, 4, 16, 5, 17, 25, 18, 7, 19, 6};
__device__ __forceinline__ int hex27_at(int place) { return g_hex27_at[place]; }

// The one-dimensional quadratic functions p[3 axis + i] and their derivatives.
__device__ __forceinline__ void hex27_axes(const double* xi, double* p, double* d) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double x = xi[a], h = 0.5 * x;
    p[3 * a] = h * x - h;
    p[3 * a + 1] = 1.0 - x * x;
    p[3 * a + 2] = h * x + h;
    d[3 * a] = x - 0.5;
    d[3 * a + 1] = -2.0 * x;
    d[3 * a + 2] = x + 0.5;
  }
}
// H[3 c + m] = sum over the nodes of v_c dN/dxi_m, summed axis by axis.  v: nine
// rows (j + 3 k) of ten doubles, 3 i + c, 16-byte aligned.
__device__ __forceinline__ void hex27_gradient(const double* v, const double* p, const double* d, double* H) {
#pragma unroll
  for (int n = 0; n < 9; ++n) H[n] = 0.0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double A[3] = {0, 0, 0}, B[3] = {0, 0, 0}, C[3] = {0, 0, 0};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double2* r = reinterpret_cast<const double2*>(v + 10 * (j + 3 * k));
      double w[10];
#pragma unroll
      for (int n = 0; n < 5; ++n) {
        const double2 t = r[n];
        w[2 * n] = t.x;
        w[2 * n + 1] = t.y;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double s = p[0] * w[c] + p[1] * w[3 + c] + p[2] * w[6 + c];
        const double t = d[0] * w[c] + d[1] * w[3 + c] + d[2] * w[6 + c];
        A[c] += p[3 + j] * t;
        B[c] += d[3 + j] * s;
        C[c] += p[3 + j] * s;
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      H[3 * c] += p[6 + k] * A[c];
      H[3 * c + 1] += p[6 + k] * B[c];
      H[3 * c + 2] += d[6 + k] * C[c];
    }
  }
}
// Value t of the 36 half edge vectors (3 (4 axis + edge) + component) of a Hex8
// with its corners in axis order (x + 2 y + 4 z).
__device__ __forceinline__ double hex8_edge(const double* corner, int t) {
  const int axis = t / 12, ed = t / 3 % 4, c = t % 3;
  const int lo = axis == 0 ? 2 * ed : (axis == 1 ? (ed & 1) | (ed & 2) << 1 : ed);
  return 0.5 * (corner[3 * (lo + (1 << axis)) + c] - corner[3 * lo + c]);
}
// Jacobian of the trilinear geometry from them (16-byte aligned).
__device__ __forceinline__ void hex8_jacobian_edges(const double* se, const double* xi, double* J) {
  double lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = 0.5 - 0.5 * xi[a];
    hi[a] = 0.5 + 0.5 * xi[a];
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
    const double w[4] = {lo[b] * lo[c], hi[b] * lo[c], lo[b] * hi[c], hi[b] * hi[c]};
    double v[12];
    const double2* r = reinterpret_cast<const double2*>(se + 12 * a);
#pragma unroll
    for (int n = 0; n < 6; ++n) {
      const double2 t = r[n];
      v[2 * n] = t.x;
      v[2 * n + 1] = t.y;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) J[3 * i + a] = w[0] * v[i] + w[1] * v[3 + i] + w[2] * v[6 + i] + w[3] * v[9 + i];
  }
}

template <class R>
__device__ __forceinline__ R det3(const R* m) {
  return m[0] * (m[4] * m[8] - m[7] * m[5]) - m[1] * (m[3] * m[8] - m[6] * m[5]) + m[2] * (m[3] * m[7] - m[6] * m[4]);
}
// inverse (row-major), returns det; out undefined when det == 0
template <class R>
__device__ __forceinline__ R inv3(const R* m, R* o) {
  R d = det3(m);
  o[0] = (m[4] * m[8] - m[7] * m[5]) / d;
  o[1] = -(m[1] * m[8] - m[7] * m[2]) / d;
  o[2] = (m[1] * m[5] - m[4] * m[2]) / d;
  o[3] = -(m[3] * m[8] - m[6] * m[5]) / d;
  o[4] = (m[0] * m[8] - m[6] * m[2]) / d;
  o[5] = -(m[0] * m[5] - m[3] * m[2]) / d;
  o[6] = (m[3] * m[7] - m[6] * m[4]) / d;
  o[7] = -(m[0] * m[7] - m[6] * m[1]) / d;
  o[8] = (m[0] * m[4] - m[3] * m[1]) / d;
  return d;
}

// Cofactor matrix of m (= det m * m^-T) and det m, without divisions.
__device__ __forceinline__ double cofactors(const double* m, double* c) {
  c[0] = m[4] * m[8] - m[5] * m[7];
  c[1] = m[5] * m[6] - m[3] * m[8];
  c[2] = m[3] * m[7] - m[4] * m[6];
  c[3] = m[2] * m[7] - m[1] * m[8];
  c[4] = m[0] * m[8] - m[2] * m[6];
  c[5] = m[1] * m[6] - m[0] * m[7];
  c[6] = m[1] * m[5] - m[2] * m[4];
  c[7] = m[2] * m[3] - m[0] * m[5];
  c[8] = m[0] * m[4] - m[1] * m[3];
  return m[0] * c[0] + m[1] * c[1] + m[2] * c[2];
}

// ---- materials (materials.rs) -----------------------------------------------
// Per quadrature point state.  M1 / M2 are the two matrices the pair
// contraction needs: SNH: M1 = Cof(F) = J F^-T, StVK: M1 = S, M2 = F F^T.
template <class R>
struct QpState {
  R F[9];
  R M1[9];
  R M2[9];
  R s1, s2, s3, s4;
  R P[9];
};

template <class R>
__device__ __forceinline__ bool snh_state(const R* F, R mu0, R lam0, QpState<R>& q, bool need_stress) {
  const R d = R(3.0);
  R mu = (d + R(1.0)) / d * mu0;
  R lam = lam0 + (R(1.0) - R(2.0) / (d * (d + R(1.0)))) * mu0;
  R alpha = R(1.0) + mu / lam * (d / (d + R(1.0)));
  R IC = R(0.0);
#pragma unroll
  for (int k = 0; k < 9; ++k) IC += F[k] * F[k];
  R Fi[9];
  R J = inv3(F, Fi);
  if (J == R(0.0)) return false;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) q.M1[3 * i + j] = Fi[3 * j + i] * J;  // dJ/dF = F^-T J
  R beta = IC + R(1.0);
  q.s1 = mu * (R(1.0) - R(1.0) / beta);
  q.s2 = mu * R(2.0) / (beta * beta);
  q.s3 = lam * (J - alpha);
  q.s4 = lam;
  if (need_stress) {
    R cf = mu * (R(1.0) - R(1.0) / (IC + R(1.0))), cj = lam * (J - alpha);
#pragma unroll
    for (int k = 0; k < 9; ++k) q.P[k] = F[k] * cf + q.M1[k] * cj;
  }
  return true;
}

template <class R>
__device__ __forceinline__ void stvk_state(const R* F, R mu, R lam, QpState<R>& q, bool need_stress) {
  R E[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R s = F[i] * F[j] + F[3 + i] * F[3 + j] + F[6 + i] * F[6 + j];  // (F^T F)(i,j)
      E[3 * i + j] = (s - (i == j ? R(1.0) : R(0.0))) * R(0.5);
    }
  R tr = E[0] + E[4] + E[8];
#pragma unroll
  for (int k = 0; k < 9; ++k) q.M1[k] = E[k] * R(2.0) * mu + ((k % 4 == 0) ? lam * tr : R(0.0));
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) q.M2[3 * i + j] = F[3 * i] * F[3 * j] + F[3 * i + 1] * F[3 * j + 1] + F[3 * i + 2] * F[3 * j + 2];
  q.s1 = mu;
  q.s4 = lam;
  if (need_stress) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        q.P[3 * i + j] = F[3 * i] * q.M1[j] + F[3 * i + 1] * q.M1[3 + j] + F[3 * i + 2] * q.M1[6 + j];
  }
}

template <class R>
__device__ __forceinline__ bool material_state(int kind, const R* F, R mu, R lam, QpState<R>& q,
                                               bool need_stress) {
#pragma unroll
  for (int k = 0; k < 9; ++k) q.F[k] = F[k];
  if (kind == HOEFEM_MAT_SNH) return snh_state(F, mu, lam, q, need_stress);
  stvk_state(F, mu, lam, q, need_stress);
  return true;
}

template <class R>
__device__ __forceinline__ void mat3vec(const R* M, const R* a, R* o) {
  o[0] = M[0] * a[0] + M[1] * a[1] + M[2] * a[2];
  o[1] = M[3] * a[0] + M[4] * a[1] + M[5] * a[2];
  o[2] = M[6] * a[0] + M[7] * a[1] + M[8] * a[2];
}

// Per quadrature point data the pair contraction needs (13 values): T = F
// (SNH, cross term) or F F^T (StVK), and four scalars (SNH: s1, s2, s3 =
// lam (J - alpha), s4 = lam; StVK: s1 = mu, s4 = lam).
template <class R>
struct QpPair {
  R T[9];
  R s1, s2, s3, s4;
};

template <class R>
__device__ __forceinline__ void qp_pair_from(int kind, const QpState<R>& q, QpPair<R>& o) {
#pragma unroll
  for (int k = 0; k < 9; ++k) o.T[k] = (kind == HOEFEM_MAT_SNH) ? q.F[k] : q.M2[k];
  o.s1 = q.s1;
  o.s2 = q.s2;
  o.s3 = q.s3;
  o.s4 = q.s4;
}

// What the pair contraction needs of a point (material_state of
// element_math.cuh without the stress): the stable Neo-Hookean Cof F comes from
// the minors instead of det F * F^-T, which takes nine FP64 divisions.
// Returns false where F is doubtful (below).
__device__ __forceinline__ bool det_doubtful(double det, const double* cof, double scale);
__device__ __forceinline__ bool point_state(int kind, const double* F, double mu0, double lam0, QpPair<double>& o,
                                            double* M1) {
  if (kind == HOEFEM_MAT_SNH) {
    const double mu = 4.0 / 3.0 * mu0, lam = lam0 + (1.0 - 2.0 / 12.0) * mu0;
    const double alpha = 1.0 + mu / lam * 0.75;
    double IC = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      IC += F[k] * F[k];
      o.T[k] = F[k];
    }
    const double J = cofactors(F, M1);
    const double ib = 1.0 / (IC + 1.0);
    o.s1 = mu * (1.0 - ib);
    o.s2 = mu * 2.0 * ib * ib;
    o.s3 = lam * (J - alpha);
    o.s4 = lam;
    return !det_doubtful(J, M1, 1.0);
  }
  QpState<double> st;
  stvk_state(F, mu0, lam0, st, false);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    o.T[k] = st.M2[k];
    M1[k] = st.M1[k];
  }
  o.s1 = st.s1;
  o.s4 = st.s4;
  o.s2 = o.s3 = 0.0;
  return true;
}

// ---- singular points ---------------------------------------------------------
// A point is singular when the determinant of its Jacobian, or of F for the
// stable Neo-Hookean material, is exactly zero in the node sums of the colored
// kernels.  The faster kernels form both in another order, so a determinant that
// is zero there may be a rounding residue here: they ask whether it is zero to
// rounding (det_doubtful, m of order scale), and only such points are evaluated
// again as those sums (tet10_singular, hex27_singular).
__device__ __forceinline__ bool det_doubtful(double det, const double* cof, double scale) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 9; ++k) s += fabs(cof[k]);
  return !(fabs(det) > 1e-10 * s * scale);
}
// corner: 4 x 3, un: 10 x 3.
__device__ __noinline__ bool tet10_singular(int kind, const double* corner, const double* un, const double* point) {
  const double xi[3] = {point[0], point[1], point[2]};
  double J[9], Ji[9], F[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  tet4_jacobian(corner, J);
  if (inv3(J, Ji) == 0.0) return true;
  if (kind != HOEFEM_MAT_SNH) return false;
#pragma unroll 1
  for (int I = 0; I < 10; ++I) {
    double gr[3], G[3];
    tet10_grad(I, xi, gr);
    for (int k = 0; k < 3; ++k) G[k] = Ji[k] * gr[0] + Ji[3 + k] * gr[1] + Ji[6 + k] * gr[2];
    for (int c = 0; c < 3; ++c)
      for (int k = 0; k < 3; ++k) F[3 * c + k] += un[3 * I + c] * G[k];
  }
  F[0] += 1.0;
  F[4] += 1.0;
  F[8] += 1.0;
  return det3(F) == 0.0;
}
// corner: 8 x 3 and un (nine rows of ten), both in axis order.
__device__ __noinline__ bool hex27_singular(int kind, const double* corner, const double* un, const double* point) {
  const double xi[3] = {point[0], point[1], point[2]};
  double Xc[24], J[9], Ji[9], F[9];
#pragma unroll 1
  for (int I = 0; I < 8; ++I) {
    const signed char* a = c_hex27_alpha[I];
    for (int k = 0; k < 3; ++k) Xc[3 * I + k] = corner[3 * ((a[0] > 0) + 2 * (a[1] > 0) + 4 * (a[2] > 0)) + k];
  }
  hex8_jacobian(Xc, xi, J);
  if (inv3(J, Ji) == 0.0) return true;
  if (kind != HOEFEM_MAT_SNH) return false;
#pragma unroll 1
  for (int n = 0; n < 9; ++n) {  // a warp's sum over its lanes, lane = node
    const int c = n / 3, k = n - 3 * c;
    double t[32];
#pragma unroll 1
    for (int I = 0; I < 32; ++I) {
      t[I] = 0.0;
      if (I >= 27) continue;
      const signed char* a = c_hex27_alpha[I];
      double gr[3];
      hex27_grad(I, xi, gr);
      const double G = Ji[k] * gr[0] + Ji[3 + k] * gr[1] + Ji[6 + k] * gr[2];
      t[I] = __dmul_rn(un[10 * (a[1] + 1 + 3 * (a[2] + 1)) + 3 * (a[0] + 1) + c], G);
    }
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1)
      for (int I = 0; I < o; ++I) t[I] += t[I + o];
    F[n] = t[0] + (c == k ? 1.0 : 0.0);
  }
  return det3(F) == 0.0;
}

// Stiffness block of node pair (I row, J column), added into acc (3x3 row-major).
// Per-node vectors: v[0..2] = a, v[3..5] = F a, v[6..8] = M1 a.
//  SNH : s1 (aI.aJ) I + s2 (F aI)(F aJ)^T + lam (Cof aI)(Cof aJ)^T + s3 eps_ijm (F (aI x aJ))_m
//  StVK: (aJ . S aI) I + mu (F aJ)(F aI)^T + mu (aI.aJ) F F^T + lam (F aI)(F aJ)^T
template <class R>
__device__ __forceinline__ void pair_block(int kind, const QpPair<R>& q, const R* vI, const R* vJ, R* acc) {
  R dot = vI[0] * vJ[0] + vI[1] * vJ[1] + vI[2] * vJ[2];
  if (kind == HOEFEM_MAT_SNH) {
    R cr[3] = {vI[1] * vJ[2] - vI[2] * vJ[1], vI[2] * vJ[0] - vI[0] * vJ[2], vI[0] * vJ[1] - vI[1] * vJ[0]};
    R w[3];
    mat3vec(q.T, cr, w);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[3 * i + j] += q.s2 * vI[3 + i] * vJ[3 + j] + q.s4 * vI[6 + i] * vJ[6 + j];
    R d1 = q.s1 * dot;
    acc[0] += d1; acc[4] += d1; acc[8] += d1;
    // eps_ijm w_m: (0,1)=w2 (0,2)=-w1 (1,0)=-w2 (1,2)=w0 (2,0)=w1 (2,1)=-w0
    R s3 = q.s3;
    acc[1] += s3 * w[2]; acc[2] -= s3 * w[1];
    acc[3] -= s3 * w[2]; acc[5] += s3 * w[0];
    acc[6] += s3 * w[1]; acc[7] -= s3 * w[0];
  } else {
    R d0 = vJ[0] * vI[6] + vJ[1] * vI[7] + vJ[2] * vI[8];  // aJ . S aI
    R mu = q.s1, lam = q.s4;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        acc[3 * i + j] += mu * vJ[3 + i] * vI[3 + j] + mu * dot * q.T[3 * i + j] + lam * vI[3 + i] * vJ[3 + j];
    acc[0] += d0; acc[4] += d0; acc[8] += d0;
  }
}

__device__ __forceinline__ void quad_rule(const BlockDev& b, int e, int& q0, int& nq) {
  if (b.uniform) { q0 = 0; nq = b.nq; }
  else { q0 = b.qoff[e]; nq = b.qoff[e + 1] - q0; }
}

}  // namespace
}  // namespace hoefem
