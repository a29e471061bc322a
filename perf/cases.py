"""Performance cases of the per-step path: element assembly, Schwarz
preconditioner, conjugate gradient, whole backward-Euler Newton steps (one
scene and batched) and the embedded quadrature construction, each through the
package's public entry points.

  listed()            the cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call
  run(state)          one pass, returning its outputs
  work(case)          bytes and operations one pass cannot do without
  exact(case, seed)   the outputs in 64-bit arithmetic by plain torch

Meshes: "tet" is a box of nx x ny x nz cells of size h = 0.025 or 1 / cells,
6 Tet10 each, stable Neo-Hookean (E = 1e6, nu = 0.4); "cylinder" is the Hex27
background grid of n^3 cells clipped to a hollow cylinder, with one quadrature
rule per cut cell, St. Venant-Kirchhoff (E = 5e5, nu = 0.45).
"""
import math

import numpy as np
import torch

import higher_order_embedded_fem_b200 as H

DT = 1e-3
DENSITY = 1000.0
GRAVITY = -9.81
# Tight linear solves, so that what a solve or a step returns does not hang on
# the iteration at which the CG stopped.
CG_TOL = 1e-10
CG_MAX = 5000
DELTA = 1e-3  # the integrator's residual-replacement threshold
BATCH_SCENES = 64


def listed():
    return [
        # explicit stepping or a residual check on a small scene: launch latency
        {"name": "forces_tet_small", "kind": "forces", "mesh": "tet", "nx": 8, "ny": 8, "nz": 8},
        # the residual of the embedded cylinder, evaluated in every line-search trial
        {"name": "forces_cylinder", "kind": "forces", "mesh": "cylinder", "n": 24},
        # tangent assembly of the large Tet10 box (201,600 elements, 70.9 M non-zeros)
        {"name": "stiffness_tet_large", "kind": "stiffness", "mesh": "tet", "nx": 40, "ny": 40, "nz": 21, "mixed": False},
        # the same with FP32 element arithmetic at an ordinary, odd size
        {"name": "stiffness_tet_mixed", "kind": "stiffness", "mesh": "tet", "nx": 23, "ny": 19, "nz": 21, "mixed": True},
        # tangent assembly of the embedded cylinder, a rule of its own in every cut cell
        {"name": "stiffness_cylinder", "kind": "stiffness", "mesh": "cylinder", "n": 24, "mixed": False},
        # the preconditioner of one Newton iteration: invert every subdomain block, apply once
        {"name": "schwarz_cylinder", "kind": "schwarz", "mesh": "cylinder", "n": 24},
        # one Schwarz-preconditioned solve with a program's own matrix
        {"name": "cg_cylinder", "kind": "cg", "mesh": "cylinder", "n": 24, "mixed": False},
        # one diagonally preconditioned mixed-precision solve, odd grid
        {"name": "cg_tet_mixed", "kind": "cg", "mesh": "tet", "nx": 31, "ny": 29, "nz": 17, "mixed": True},
        # interactive step of a small scene
        {"name": "newton_tet_small", "kind": "newton", "mesh": "tet", "nx": 8, "ny": 8, "nz": 8, "mixed": False},
        # the benchmark's step: embedded cylinder, mixed precision
        {"name": "newton_cylinder_mixed", "kind": "newton", "mesh": "cylinder", "n": 24, "mixed": True},
        # many small scenes in one step (parameter studies, data generation)
        {"name": "newton_batch", "kind": "batch", "scenes": BATCH_SCENES, "low": 200, "high": 2000},
        # scene set-up: cut the background grid, build and simplify the cut-cell rules
        {"name": "embed_cylinder", "kind": "embed", "n": 24, "nr": 3, "ntheta": 144, "nz": 72},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo, hi):
    """A box of roughly log-uniform cell count in [lo, hi], any three sides."""
    cells = _log(rng, lo, hi)
    a, b = math.exp(rng.uniform(-0.4, 0.4)), math.exp(rng.uniform(-0.4, 0.4))
    n = cells ** (1.0 / 3.0)
    nx, ny = max(1, round(n * a)), max(1, round(n * b))
    return {"mesh": "tet", "nx": nx, "ny": ny, "nz": max(1, min(round(cells / (nx * ny)), int(hi) // (nx * ny)))}


def draw(rng):
    kind = rng.choice(["forces", "stiffness", "schwarz", "cg", "newton", "batch", "embed"])
    mixed = rng.random() < 0.5
    if kind == "batch":
        low = round(_log(rng, 20, 400))
        return {"kind": "batch", "scenes": rng.randint(5, BATCH_SCENES), "low": low, "high": rng.randint(2 * low, 2000)}
    if kind == "embed":
        n = rng.randint(5, 24)
        return {"kind": "embed", "n": n, "nr": rng.randint(1, 3), "ntheta": rng.randint(24, 6 * n), "nz": rng.randint(6, 3 * n)}
    if kind == "schwarz" or rng.random() < 0.5:
        c = {"mesh": "cylinder", "n": rng.randint(6, 24)}
    else:
        # whole steps and solves up to the size of the listed solve
        c = _box(rng, 30, 33600 if kind in ("forces", "stiffness") else 15283)
    if kind in ("stiffness", "cg", "newton"):
        c["mixed"] = mixed
    return {"kind": kind, **c}


# ---- inputs -------------------------------------------------------------------

def _mesh(case):
    """(vertices, blocks, cell size, volume fractions): the scene's arrays."""
    if case["mesh"] == "cylinder":
        return H.scenes.embedded_cylinder(case["n"], 0.3, 0.4, 8, 27, 2)
    return H.scenes.tet10_box(_cell(case), case["nx"], case["ny"], case["nz"], 1)


def _cell(case):
    return 1.0 / case["nx"] if max(case["nx"], case["ny"], case["nz"]) <= 8 else 0.025


def _lame(case):
    young, nu = (5e5, 0.45) if case["mesh"] == "cylinder" else (1e6, 0.4)
    mu = 0.5 * young / (1.0 + nu)
    return mu, 0.5 * mu * nu / (1.0 - 2.0 * nu)


def _displacement(case, scene, seed):
    """Smooth sway plus noise (cylinder) or noise (box), the kinds of state the
    benchmark steps from.  The cylinder's noise stays small enough for the
    Jacobian of its thinly cut cells to remain positive definite at any seed."""
    rng = np.random.default_rng(seed)
    X = scene.vertices
    h = scene.cell_size
    u = np.zeros_like(X)
    if case["mesh"] == "cylinder":
        u[:, 0] = 0.02 * X[:, 2] ** 2
        u[:, 1] = 0.01 * X[:, 2] ** 2
        u += rng.normal(0.0, 0.0001 * h, X.shape)
    else:
        u += rng.normal(0.0, 0.02 * h, X.shape)
    return u.reshape(-1)


def _rhs(ndof, bc, seed):
    b = np.random.default_rng(seed + 1).normal(0.0, 1.0, ndof)
    b.reshape(-1, 3)[bc] = 0.0
    return b


def _model(case, scene):
    if case["mesh"] == "cylinder":
        b0, b1 = scene.blocks
        m = H.EmbeddedModel3d(scene.vertices, b0.connectivity, b1.connectivity, (b0.weights, b0.points),
                              (b1.offsets, b1.weights, b1.points))
        mat = H.StVKMaterial(H.LameParameters(*_lame(case)))
    else:
        b = scene.blocks[0]
        m = H.NodalModel3d(scene.vertices, b.connectivity, (b.weights, b.points))
        mat = H.StableNeoHookeanMaterial(H.LameParameters(*_lame(case)))
    return m, mat


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _schwarz(model, scene):
    return H.SchwarzPreconditionerComponent.from_embedded_model(model, scene.volume_fractions, 0.5).build(model)


def _bottom(scene):
    return np.nonzero(scene.vertices[:, 2] <= 1e-9)[0].astype(np.int64)


def _batch_specs(case, seed):
    """Scenes of the batch: sizes from the case alone, materials and states from the seed."""
    size = np.random.default_rng(1234)
    rng = np.random.default_rng(seed)
    specs = []
    for k in range(case["scenes"]):
        target = math.exp(size.uniform(math.log(case["low"]), math.log(case["high"])))
        tet = k % 2 == 0
        cells = max(1.0, target / 6.0 if tet else target)
        n = max(1, round(cells ** (1.0 / 3.0)))
        nz = max(1, round(cells / (n * n)))
        specs.append({"tet": tet, "n": n, "nz": nz, "h": 1.0 / max(n, nz),
                      "young": math.exp(rng.uniform(math.log(1e5), math.log(1e7))), "nu": rng.uniform(0.3, 0.48),
                      "sway": 0.01 * rng.uniform(-1.0, 1.0, 2), "noise": int(rng.integers(1 << 30))})
    return specs


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "embed":
        bg = H.scenes.hex27_box(1.0, 1, 1, 1, case["n"])
        X, T = H.scenes.hollow_cylinder_tets(0.3, 0.4, 1.0, case["nr"], case["ntheta"], case["nz"])
        # off the grid's symmetry planes; every seed moves the vertices a little, which
        # keeps the set of cut cells (and the outputs' lengths)
        X = X + np.array([0.0123, -0.0077, 0.0]) + np.random.default_rng(seed).uniform(-1e-7, 1e-7, X.shape)
        st.update(V=bg.vertices, C=bg.blocks[0].connectivity, X=X, T=T,
                  interior=(bg.blocks[0].weights, bg.blocks[0].points), tet=H.tet_quadrature_strength(3))
        return st
    st["stream"] = torch.cuda.Stream()
    handle = st["stream"].cuda_stream
    if kind == "batch":
        models, mats, bcs, us = [], [], [], []
        for s in _batch_specs(case, seed):
            scene = (H.scenes.tet10_box if s["tet"] else H.scenes.hex27_box)(s["h"], s["n"], s["n"], s["nz"], 1)
            b = scene.blocks[0]
            models.append(H.NodalModel3d(scene.vertices, b.connectivity, (b.weights, b.points), b.kind))
            mats.append(H.StableNeoHookeanMaterial(H.YoungPoisson(s["young"], s["nu"])))
            bcs.append(_bottom(scene))
            u = np.random.default_rng(s["noise"]).normal(0.0, 0.001 * scene.cell_size, scene.vertices.shape)
            u[:, :2] += s["sway"] * scene.vertices[:, 2:] ** 2
            us.append(u.reshape(-1))
        B = H.BatchedNewtonCgIntegrator3d(models, mats, DENSITY, bcs)
        B.set_tolerances(CG_TOL, CG_MAX, 100)
        B.set_stream(handle)
        u0 = _cuda(np.concatenate(us))
        st.update(integ=B, u0=u0, v0=torch.zeros_like(u0), u=u0.clone(), v=torch.zeros_like(u0))
        torch.cuda.synchronize()
        return st
    scene = _mesh(case)
    m, mat = _model(case, scene)
    m.set_stream(handle)
    u = _cuda(_displacement(case, scene, seed))
    bc = _bottom(scene)
    st.update(model=m, mat=mat, u0=u)
    if kind == "stiffness":
        st["values"] = torch.empty(m.nnz, dtype=torch.float64, device="cuda")
    if kind in ("schwarz", "cg"):
        # the matrix of one Newton iteration, dt^2 K(u) + M with the bottom clamped
        K, M = (torch.zeros(m.nnz, dtype=torch.float64, device="cuda") for _ in range(2))
        J = torch.empty_like(K)
        torch.cuda.synchronize()
        m.assemble_stiffness_into_par(K, u, mat)
        m.assemble_mass_into(M, DENSITY)
        m.jacobian_combination(J, DT * DT, K, 1.0, M, bc)
        st.update(J=J, b=_cuda(_rhs(m.ndof(), bc, seed)), out=torch.zeros_like(u))
        st["P"] = _schwarz(m, scene) if case["mesh"] == "cylinder" else H.DiagonalPreconditioner(m)
        if kind == "cg":
            st["P"].update(J)
            st["solver"] = (H.ConjugateGradient(m).with_operator(J).with_preconditioner(st["P"])
                            .with_stopping_criterion(H.RelativeResidualCriterion(CG_TOL)).with_max_iter(CG_MAX))
    if kind == "newton":
        P = _schwarz(m, scene) if case["mesh"] == "cylinder" else None
        it = H.NewtonCgIntegrator3d(m, mat, DENSITY, bc, GRAVITY, True, P)
        it.set_tolerances(CG_TOL, CG_MAX, 100)
        it.set_precision(case["mixed"], DELTA)
        st.update(integ=it, v0=torch.zeros_like(u), u=u.clone(), v=torch.zeros_like(u))
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind == "embed":
        emb = H.embed_mesh_3d(st["V"], st["C"], st["X"], st["T"])
        quad = H.embed_quadrature_3d(emb, st["interior"], st["tet"]).simplified(3)
        return {"class": emb.cell_class, "volume": emb.cut_volume, "offsets": quad.offsets, "weights": quad.weights,
                "points": quad.points}
    with torch.cuda.stream(st["stream"]):
        if kind == "forces":
            return st["model"].assemble_elastic_pseudo_forces(st["u0"], st["mat"])
        if kind == "stiffness":
            return st["model"].assemble_stiffness_into_precision(st["values"].zero_(), st["u0"], st["mat"],
                                                                 st["case"]["mixed"])
        if kind == "schwarz":
            st["P"].update(st["J"])
            return st["P"].apply(st["b"], st["out"])
        if kind == "cg":
            x = st["out"].zero_()
            if st["case"]["mixed"]:
                st["solver"].solve_with_guess_mixed(st["b"], x, DELTA)
            else:
                st["solver"].solve_with_guess(st["b"], x)
            return x
        u, v = st["u"].copy_(st["u0"]), st["v"].copy_(st["v0"])
        st["integ"].step(u, v, 0.0, DT)
        return {"u": u, "v": v}


# ---- work ---------------------------------------------------------------------

def _sizes(case):
    """(nodes, stored matrix entries, elements, nodes per element, points per element, subdomains)."""
    if case["mesh"] == "cylinder":
        # cells the shell 0.3 <= r <= 0.4 touches: 0.3 of the grid at n = 24, about
        # 10.3 nodes a cell and 168 entries a row
        ne = int(0.31 * case["n"] ** 3)
        nv = int(10.3 * ne)
        return nv, 9 * 56 * nv, ne, 27, 20, int(0.125 * case["n"] ** 3)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nv = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    return nv, 9 * 28 * nv, 6 * nx * ny * nz, 10, 14, 0


def work(case):
    kind = case["kind"]
    if kind == "embed":
        # every tet against the few cells it meets, 4 tets a cut cell piece, 4 points each
        tets = 6 * case["nr"] * case["ntheta"] * case["nz"]
        pts = 45 * tets
        return {"bytes": 32 * tets + 216 * case["n"] ** 3 + 2 * 32 * 20 * case["n"] ** 2, "flops": 20 * 20 * 2 * pts}
    if kind == "batch":
        each = 0.5 * (case["low"] + case["high"])
        nv, nnz, ne, nn, nq, nsub = int(case["scenes"] * each * 4), 0, int(case["scenes"] * each), 27, 14, 0
        nnz = 9 * 40 * nv
    else:
        nv, nnz, ne, nn, nq, nsub = _sizes(case)
    vec = 24 * nv
    element = 4 * nn * ne + 32 * nq * (1 if case.get("mesh") == "tet" else ne)
    force = ne * nq * (36 * nn + 200)
    tangent = ne * nq * (nn * (nn + 1) // 2 * 120 + 60 * nn)
    if kind == "forces":
        return {"bytes": 3 * vec + element, "flops": force}
    if kind == "stiffness":
        return {"bytes": 2 * vec + element + 8 * nnz, "flops": tangent}
    if kind == "schwarz":
        return {"bytes": 2 * vec + 8 * nnz, "flops": nsub * 2 * 81 ** 3}
    value = 4 if case.get("mixed") else 8
    if kind == "cg":
        # the matrix once and, for the products, 80 iterations at least
        return {"bytes": 2 * vec + value * nnz, "flops": 80 * 2 * (nnz + 6561 * nsub)}
    # a step: states in and out; 3 Newton iterations of 50 CG iterations at least
    return {"bytes": 4 * vec + element, "flops": 3 * (tangent + force + 50 * 2 * (nnz + 6561 * nsub))}


# ---- the outputs in 64-bit arithmetic -------------------------------------------

_EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (2, 3), (1, 3))
_HEX = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1),
        (0, -1, -1), (-1, 0, -1), (-1, -1, 0), (1, 0, -1), (1, -1, 0), (0, 1, -1), (1, 1, 0), (-1, 1, 0),
        (0, -1, 1), (-1, 0, 1), (1, 0, 1), (0, 1, 1), (0, 0, -1), (0, -1, 0), (-1, 0, 0), (1, 0, 0),
        (0, 1, 0), (0, 0, 1), (0, 0, 0))


def _basis(nn, xi):
    """Shape functions (.., nn), their reference gradients (.., nn, 3) and the
    gradients of the vertex basis that maps the geometry (.., nc, 3)."""
    one = torch.ones_like(xi[..., 0])
    if nn == 10:
        p = torch.stack([-0.5 * (xi.sum(-1) + 1.0)] + [0.5 * (xi[..., k] + 1.0) for k in range(3)], -1)
        g = 0.5 * torch.tensor([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=xi.dtype, device=xi.device)
        phi = [p[..., a] * (2 * p[..., a] - 1) for a in range(4)] + [4 * p[..., a] * p[..., b] for a, b in _EDGES]
        dphi = [(4 * p[..., a, None] - 1) * g[a] for a in range(4)]
        dphi += [4 * (p[..., a, None] * g[b] + p[..., b, None] * g[a]) for a, b in _EDGES]
        return torch.stack(phi, -1), torch.stack(dphi, -2), g.expand(*xi.shape[:-1], 4, 3)
    # one-dimensional quadratics at -1, 0, 1 and their derivatives
    q = {-1: 0.5 * xi * (xi - 1), 0: 1 - xi * xi, 1: 0.5 * xi * (xi + 1)}
    dq = {-1: xi - 0.5, 0: -2 * xi, 1: xi + 0.5}
    li = {-1: 0.5 * (1 - xi), 1: 0.5 * (1 + xi)}
    phi, dphi, dgeo = [], [], []
    for a in _HEX:
        f = [q[a[k]][..., k] for k in range(3)]
        d = [dq[a[k]][..., k] for k in range(3)]
        phi.append(f[0] * f[1] * f[2])
        dphi.append(torch.stack([d[0] * f[1] * f[2], f[0] * d[1] * f[2], f[0] * f[1] * d[2]], -1))
    for a in _HEX[:8]:
        f = [li[a[k]][..., k] for k in range(3)]
        dgeo.append(torch.stack([0.5 * a[0] * f[1] * f[2], 0.5 * a[1] * f[0] * f[2], 0.5 * a[2] * f[0] * f[1]], -1) *
                    one[..., None])
    return torch.stack(phi, -1), torch.stack(dphi, -2), torch.stack(dgeo, -2)


class _Reference:
    """Assembly and solves of one scene in plain torch, 64 bits, on the GPU.
    Matrices are (pairs, 3, 3) node blocks in ascending (row, column) order."""

    def __init__(self, case, scene):
        self.snh = case["mesh"] == "tet"
        self.mu, self.lam = _lame(case)
        self.X = _cuda(scene.vertices)
        self.nv = len(scene.vertices)
        self.blocks = []
        keys = torch.empty(0, dtype=torch.int64, device="cuda")
        for b in scene.blocks:
            conn, w, p = _cuda(b.connectivity), _cuda(b.weights), _cuda(b.points)
            ne, nn = conn.shape
            if b.offsets is None:
                wq, pq = w.expand(ne, -1), p.expand(ne, -1, -1)
            else:
                # pad every rule to the longest with points of weight zero
                off = _cuda(b.offsets)
                k = torch.arange(int((off[1:] - off[:-1]).max()), device="cuda")
                at = off[:-1, None] + k
                inside = at < off[1:, None]
                at = torch.where(inside, at, off[:-1, None])
                wq, pq = torch.where(inside, w[at], torch.zeros_like(w[:1])), p[at]
            self.blocks.append((conn, wq, pq))
            pair = (conn[:, :, None] * self.nv + conn[:, None, :]).reshape(-1)
            keys = torch.unique(torch.cat([keys, torch.unique(pair)]))
        self.keys = keys
        self.row, self.col = keys // self.nv, keys % self.nv
        deg = torch.bincount(self.row, minlength=self.nv)
        self.off = torch.cat([deg.new_zeros(1), deg.cumsum(0)])
        self.diag = torch.searchsorted(keys, torch.arange(self.nv, device="cuda") * (self.nv + 1))

    def _chunks(self, limit=6000):
        for conn, wq, pq in self.blocks:
            for e in range(0, len(conn), limit):
                c, w, p = conn[e:e + limit], wq[e:e + limit], pq[e:e + limit]
                phi, dphi, dgeo = _basis(c.shape[1], p)
                J = torch.einsum("eci,eqck->eqik", self.X[c[:, :dgeo.shape[-2]]], dgeo)
                G = dphi @ torch.linalg.inv(J)
                yield c, w * torch.linalg.det(J).abs(), phi, G

    def _gradient(self, c, G, u):
        return torch.einsum("eni,eqnk->eqik", u.reshape(-1, 3)[c], G) + torch.eye(3, dtype=u.dtype, device=u.device)

    def _snh(self, F):
        mu = 4.0 / 3.0 * self.mu
        lam = self.lam + 5.0 / 6.0 * self.mu
        det = torch.linalg.det(F)[..., None, None]
        cof = det * torch.linalg.inv(F).transpose(-1, -2)
        return mu, lam, 1.0 + (F * F).sum((-1, -2))[..., None, None], cof, lam * (det - 1.0 - 0.75 * mu / lam)

    def _stress(self, F):
        if self.snh:
            mu, _, beta, cof, pressure = self._snh(F)
            return mu * (1.0 - 1.0 / beta) * F + pressure * cof
        return F @ self._second(F)

    def _second(self, F):
        E = 0.5 * (F.transpose(-1, -2) @ F - torch.eye(3, dtype=F.dtype, device=F.device))
        tr = E.diagonal(dim1=-1, dim2=-2).sum(-1)[..., None, None]
        return 2.0 * self.mu * E + self.lam * tr * torch.eye(3, dtype=F.dtype, device=F.device)

    def _tangent(self, F):
        """dP_ij / dF_kl as (.., 3, 3, 3, 3)."""
        eye = torch.eye(3, dtype=F.dtype, device=F.device)
        if self.snh:
            mu, lam, beta, cof, pressure = self._snh(F)
            beta, pressure = beta[..., None, None], pressure[..., None, None]
            eps = torch.zeros(3, 3, 3, dtype=F.dtype, device=F.device)
            for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
                eps[i, j, k], eps[i, k, j] = 1.0, -1.0
            dcof = torch.einsum("ikm,jln,...mn->...ijkl", eps, eps, F)
            return (mu * (1.0 - 1.0 / beta) * torch.einsum("ik,jl->ijkl", eye, eye) +
                    2.0 * mu / beta ** 2 * torch.einsum("...ij,...kl->...ijkl", F, F) +
                    lam * torch.einsum("...ij,...kl->...ijkl", cof, cof) + pressure * dcof)
        return (torch.einsum("ik,...lj->...ijkl", eye, self._second(F)) +
                self.mu * torch.einsum("...il,...kj->...ijkl", F, F) +
                self.mu * torch.einsum("...im,...km,jl->...ijkl", F, F, eye) +
                self.lam * torch.einsum("...ij,...kl->...ijkl", F, F))

    def forces(self, u):
        f = torch.zeros(self.nv, 3, dtype=u.dtype, device=u.device)
        for c, w, _, G in self._chunks():
            P = self._stress(self._gradient(c, G, u)) * w[..., None, None]
            f.index_add_(0, c.reshape(-1), -torch.einsum("eqij,eqnj->eni", P, G).reshape(-1, 3))
        return f.reshape(-1)

    def _add(self, out, c, ke):
        at = torch.searchsorted(self.keys, (c[:, :, None] * self.nv + c[:, None, :]).reshape(-1))
        out.index_add_(0, at, ke.reshape(-1, 3, 3))

    def stiffness(self, u):
        out = torch.zeros(len(self.keys), 3, 3, dtype=u.dtype, device=u.device)
        for c, w, _, G in self._chunks():
            A = (self._tangent(self._gradient(c, G, u)) * w[..., None, None, None, None]).flatten(0, 1)
            g = G.flatten(0, 1)
            n = g.shape[1]
            half = torch.matmul(A.permute(0, 1, 3, 4, 2).reshape(len(g), 27, 3), g.transpose(1, 2))  # (i k l), n
            half = half.reshape(len(g), 3, 3, 3, n).permute(0, 4, 1, 2, 3).reshape(len(g), n * 9, 3)
            ke = torch.matmul(half, g.transpose(1, 2)).reshape(len(c), -1, n, 3, 3, n).sum(1)
            self._add(out, c, ke.permute(0, 1, 4, 2, 3))
        return out

    def mass(self):
        out = torch.zeros(len(self.keys), 3, 3, dtype=torch.float64, device="cuda")
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        for c, w, phi, _ in self._chunks():
            me = DENSITY * torch.einsum("eq,eqm,eqn->emn", w, phi, phi)
            self._add(out, c, me[..., None, None] * eye)
        return out

    def clamp(self, A, bc):
        """Clamped rows and columns zero, their diagonal the first non-zero diagonal entry."""
        d = A[self.diag].diagonal(dim1=1, dim2=2).reshape(-1)
        scale = d[torch.nonzero(d)[0, 0]].abs()
        held = torch.zeros(self.nv, dtype=torch.bool, device="cuda")
        held[bc] = True
        A = torch.where((held[self.row] | held[self.col])[:, None, None], torch.zeros_like(A[:1]), A)
        A[self.diag[held]] = scale * torch.eye(3, dtype=A.dtype, device=A.device)
        return A

    def scalar(self, A):
        """The scalar CSR values: rows 3a + i, columns ascending."""
        k = torch.arange(len(A), device="cuda")
        o, d = self.off[self.row], (self.off[1:] - self.off[:-1])[self.row]
        i = torch.arange(3, device="cuda")
        at = 9 * o[:, None, None] + 3 * (d[:, None] * i)[:, :, None] + 3 * (k - o)[:, None, None] + i
        out = torch.empty(A.numel(), dtype=A.dtype, device=A.device)
        out[at.reshape(-1)] = A.reshape(-1)
        return out

    def matrix(self, A):
        deg = 3 * (self.off[1:] - self.off[:-1])
        crow = torch.cat([deg.new_zeros(1), deg.repeat_interleave(3).cumsum(0)])
        i = torch.arange(3, device="cuda")
        cols = self.scalar((3 * self.col[:, None, None] + i).expand(-1, 3, 3).contiguous())
        return torch.sparse_csr_tensor(crow, cols, self.scalar(A), (3 * self.nv, 3 * self.nv))

    def solve(self, A, b, tol=1e-14):
        """Diagonally preconditioned CG, well past the tolerance of the timed solves."""
        S = self.matrix(A)
        d = 1.0 / A[self.diag].diagonal(dim1=1, dim2=2).reshape(-1)
        x = torch.zeros_like(b)
        for _ in range(2):  # the second pass refines on the true residual
            r = b - S @ x
            z = d * r
            p, zr = z.clone(), torch.dot(z, r)
            stop = tol * torch.linalg.norm(b)
            for k in range(8000):
                q = S @ p
                a = zr / torch.dot(p, q)
                x = x + a * p
                r = r - a * q
                if k % 20 == 19 and bool(torch.linalg.norm(r) <= stop):
                    break
                z = d * r
                zr, old = torch.dot(z, r), zr
                p = z + (zr / old) * p
        return x

    def product(self, A, x):
        return self.matrix(A) @ x


def _exact_schwarz(ref, J, scene, r):
    """Sum of the inverted subdomain blocks, the inverse diagonal on the other nodes."""
    picked = scene.blocks[1].connectivity[scene.volume_fractions <= 0.5]
    c = _cuda(picked)
    at = torch.searchsorted(ref.keys, (c[:, :, None] * ref.nv + c[:, None, :]).reshape(-1))
    n = c.shape[1]
    B = J[at].reshape(-1, n, n, 3, 3).permute(0, 1, 3, 2, 4).reshape(-1, 3 * n, 3 * n)
    rr = r.reshape(-1, 3)
    z = rr / J[ref.diag].diagonal(dim1=1, dim2=2)
    z[c.reshape(-1)] = 0.0
    y = torch.linalg.solve(B, rr[c].reshape(-1, 3 * n, 1))
    return z.index_add_(0, c.reshape(-1), y.reshape(-1, 3)).reshape(-1)


def _exact_step(ref, bc, u, v):
    """One backward-Euler step: Newton with backtracking, as the integrator stops it."""
    def held(x):
        x = x.clone()
        x.reshape(-1, 3)[bc] = 0.0
        return x

    M = ref.clamp(ref.mass(), bc)
    S = ref.matrix(M)
    ones = torch.full_like(u, math.sqrt(100.0 / 3.0))
    tol = DT * 1e-5 * torch.linalg.norm(S @ ones)
    g = torch.zeros_like(u)
    g.reshape(-1, 3)[:, 2] = GRAVITY
    g = S @ g
    u, v = held(u), held(v)
    up, w = u + DT * v, torch.zeros_like(u)

    def residual(w):
        return S @ w - DT * held(g + ref.forces(held(up + DT * w)))

    F = residual(w)
    for _ in range(100):
        if torch.linalg.norm(F) <= tol:
            break
        J = ref.clamp(DT * DT * ref.stiffness(held(up + DT * w)) + M, bc)
        dx = ref.solve(J, F, 1e-13)
        for alpha in [1.0, 0.75, 0.5] + [0.25 ** (k + 1) for k in range(8)]:
            Fa = residual(w - alpha * dx)
            if torch.dot(Fa, Fa) <= (1.0 - 1e-4 * alpha) * torch.dot(F, F):
                break
        w, F = w - alpha * dx, Fa
    v = held(v + w)
    return {"u": held(u + DT * v), "v": v}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "embed"):
        return None  # dozens of scenes one by one; a selection of points, not a number
    scene = _mesh(case)
    ref = _Reference(case, scene)
    u = _cuda(_displacement(case, scene, seed))
    bc = _cuda(_bottom(scene))
    if kind == "forces":
        return ref.forces(u)
    if kind == "stiffness":
        return ref.scalar(ref.stiffness(u))
    if kind == "newton":
        return _exact_step(ref, bc, u, torch.zeros_like(u))
    J = ref.clamp(DT * DT * ref.stiffness(u) + ref.mass(), bc)
    b = _cuda(_rhs(3 * ref.nv, bc.cpu().numpy(), seed))
    return _exact_schwarz(ref, J, scene, b) if kind == "schwarz" else ref.solve(J, b)
