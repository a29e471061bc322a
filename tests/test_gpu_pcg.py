"""The persistent CG on CSR values in place (csrc/cg_persist.cu) against the
graphs of kernel chunks (taken when the SpMV variant is pinned): every value
precision and preconditioner, at sizes where its tiles can go wrong (fewer
tiles than warps, one CTA's worth, a value array that ends inside a 16-byte
granule, nodes of no element, rows of 125 neighbours, values it does not take).

Both stop on the recurrence residual at 1e-10 ||b||; the true residual may
differ from it by rounding (1 % allowed, as in the other engines' tests) and
the solutions by the two residuals over the smallest eigenvalue: 1e-6.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-10


def tet(nx, ny, nz, extra_nodes=0):
    s = H.scenes.tet10_box(1.0 / max(nx, ny, nz), nx, ny, nz, 1)
    X = np.concatenate([s.vertices, np.full((extra_nodes, 3), 9.0)])
    b = s.blocks[0]
    return s, H.NodalModel3d(X, b.connectivity, (b.weights, b.points)), H.StableNeoHookeanMaterial(H.YoungPoisson(1e6, 0.4))


def cylinder(n):
    e = H.scenes.embedded_cylinder(n, 0.3, 0.4, 8, 27, 2)
    b0, b1 = e.blocks
    m = H.EmbeddedModel3d(e.vertices, b0.connectivity, b1.connectivity, (b0.weights, b0.points),
                          (b1.offsets, b1.weights, b1.points))
    return e, m, H.StVKMaterial(H.YoungPoisson(5e5, 0.45))


def system(s, m, mat, seed=3):
    bc = s.nodes_below(2, 1e-9)
    u = H.scenes.random_normal(seed, m.ndof(), 1e-4 * s.cell_size)
    J = m.jacobian_combination(np.zeros(m.nnz), 1e-6, m.assemble_stiffness(u, mat), 1.0, m.assemble_mass(1000.0), bc)
    b = H.scenes.random_normal(seed + 1, m.ndof(), 1.0)
    b.reshape(-1, 3)[bc] = 0.0
    return J, b


def solve(m, J, P, b, mixed, max_iter=5000, tol=TOL):
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    cg = (H.ConjugateGradient(m).with_operator(J).with_preconditioner(P)
          .with_stopping_criterion(H.RelativeResidualCriterion(tol)).with_max_iter(max_iter))
    out = cg.solve_with_guess_mixed(b, x, 1e-3) if mixed else cg.solve_with_guess(b, x)
    return x, out.num_iterations


def residual(m, J, x, b):
    y = torch.zeros_like(b)
    torch.cuda.synchronize()
    m.spmv(y, J, x)
    return float((y - b).norm() / b.norm())


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("prec", ["none", "diagonal", "schwarz"])
@pytest.mark.parametrize("scene", [("tet", 1, 1, 1), ("tet", 3, 2, 1), ("tet", 9, 7, 11), ("tet", 17, 19, 13),
                                   ("cylinder", 5), ("cylinder", 13)])
def test_persistent_matches_graphs(scene, prec, mixed):
    s, m, mat = tet(*scene[1:]) if scene[0] == "tet" else cylinder(scene[1])
    if (prec == "schwarz" and scene[0] == "tet") or (prec == "none" and scene[0] == "cylinder"):
        pytest.skip("the box has no subdomains; the cylinder needs a preconditioner (2,313 to 2,320 iterations with "
                    "the SpMV variants of the graphs at 5^3, more than 5,000 at 13^3)")
    J, b = system(s, m, mat)
    P = None
    if prec == "diagonal":
        P = H.DiagonalPreconditioner(m)
    elif prec == "schwarz":
        P = H.SchwarzPreconditionerComponent.from_embedded_model(m, s.volume_fractions, 0.5).build(m)
    Jd, bd = torch.from_numpy(J).cuda(), torch.from_numpy(b).cuda()
    if P is not None:
        P.update(Jd)
    m.set_cg_engine("chunked")
    x1, i1 = solve(m, Jd, P, bd, mixed)
    x2, i2 = solve(m, Jd, P, bd, mixed)
    assert i1 == i2 and torch.equal(x1, x2)  # deterministic
    m.set_spmv_variant(32)
    xg, ig = solve(m, Jd, P, bd, mixed)
    # FP32 products: the residual replacements fall on other iterations (checked every
    # iteration here, every eighth there)
    assert abs(i1 - ig) <= (max(4, 0.05 * ig) if mixed else 1)
    assert residual(m, Jd, x1, bd) <= 1.01 * TOL
    assert float((x1 - xg).norm() / xg.norm()) < 1e-6


def test_values_that_are_not_aligned_and_nodes_of_no_element():
    s, m, mat = tet(5, 4, 3, extra_nodes=3)
    u = H.scenes.random_normal(1, m.ndof(), 1e-4 * s.cell_size)
    K, M = m.assemble_stiffness(u, mat), m.assemble_mass(1000.0)
    J = torch.from_numpy(1e-6 * K + M).cuda()
    b = torch.from_numpy(H.scenes.random_normal(2, m.ndof(), 1.0)).cuda()
    b[-9:] = 0.0  # the rows of those nodes are empty
    m.set_cg_engine("chunked")
    x, it = solve(m, J, None, b, False)
    assert residual(m, J, x, b) <= 1.01 * TOL and torch.all(x[-9:] == 0)
    buf = torch.zeros(m.nnz + 1, dtype=torch.float64, device="cuda")
    buf[1:] = J  # 8-byte aligned: the graphs take it
    xo, io = solve(m, buf[1:], None, b, False)
    assert abs(it - io) <= 1 and float((x - xo).norm() / xo.norm()) < 1e-6


def test_sharp_residual_drop_and_error_kinds():
    # mass-dominated: the diagonal preconditioner converges in few steps, each
    # far below the last, so the sums are taken from the updated residual
    s, m, mat = tet(6, 5, 4)
    M = m.assemble_mass(1000.0)
    ro, ci = m.pattern()
    diag = np.repeat(np.arange(m.ndof()), np.diff(ro)) == ci
    D = torch.from_numpy(np.where(diag, 1.0 + np.abs(M), 0.0)).cuda()
    P = H.DiagonalPreconditioner(m)
    P.update(D)
    b = torch.from_numpy(H.scenes.random_normal(2, m.ndof(), 1.0)).cuda()
    m.set_cg_engine("chunked")
    x, it = solve(m, D, P, b, False)
    assert it == 1 and residual(m, D, x, b) <= 1e-14
    J, _ = system(s, m, mat)
    J = torch.from_numpy(J).cuda()
    for k in (0, 1, 7):
        with pytest.raises(H.SolveError) as e:
            solve(m, J, P, b, False, max_iter=k)
        assert e.value.kind == H.SolveErrorKind.MaxIterationsReached and e.value.output.num_iterations == k
    with pytest.raises(H.SolveError) as e:
        solve(m, -J, None, b, False)
    assert e.value.kind == H.SolveErrorKind.IndefiniteOperator and e.value.output.num_iterations == 0
    x, it = solve(m, J, None, torch.zeros_like(b), False)
    assert it == 0 and torch.all(x == 0)
