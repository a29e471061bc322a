"""Solves that cannot converge end in every engine, as the graphs of kernel chunks
end them: with HOEFEM_CG_MAX_ITERATIONS at the limit, which without one of the
caller's is 10 n iterations rounded up to chunks of eight, plus two chunks.

A NaN in the right-hand side or the matrix makes x a NaN everywhere after one
iteration, so the outcome of the limit is known then; the graphs run on to it and
give the same outcome.  A tolerance of 1e-17 lies below the rounding of a true
residual (2^-53 of the sums that form it), so a mixed solve's replacements keep
refuting the recurrence.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def setup(kind):
    if kind == "tet":
        s = H.scenes.tet10_box(1.0 / 3.0, 3, 2, 1, 1)
        b = s.blocks[0]
        m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points))
        mat = H.StableNeoHookeanMaterial(H.YoungPoisson(1e6, 0.4))
    else:
        s = H.scenes.embedded_cylinder(5, 0.3, 0.4, 8, 27, 2)
        b0, b1 = s.blocks
        m = H.EmbeddedModel3d(s.vertices, b0.connectivity, b1.connectivity, (b0.weights, b0.points),
                              (b1.offsets, b1.weights, b1.points))
        mat = H.StVKMaterial(H.YoungPoisson(5e5, 0.45))
    u = H.scenes.random_normal(3, m.ndof(), 1e-4 * s.cell_size)
    J = torch.from_numpy(1e-6 * m.assemble_stiffness(u, mat) + m.assemble_mass(1000.0)).cuda()
    if kind == "cylinder":
        P = H.SchwarzPreconditionerComponent.from_embedded_model(m, s.volume_fractions, 0.5).build(m)
    else:
        P = H.DiagonalPreconditioner(m)
    P.update(J)
    return m, J, P, torch.from_numpy(H.scenes.random_normal(4, m.ndof(), 1.0)).cuda()


def solve(m, J, P, b, mixed, max_iter, tol=1e-10):
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    cg = (H.ConjugateGradient(m).with_operator(J).with_preconditioner(P)
          .with_stopping_criterion(H.RelativeResidualCriterion(tol)))
    if max_iter is not None:
        cg = cg.with_max_iter(max_iter)
    with pytest.raises(H.SolveError) as e:
        cg.solve_with_guess_mixed(b, x, 1e-3) if mixed else cg.solve_with_guess(b, x)
    return x, e.value.kind, e.value.output.num_iterations


def default_limit(n):
    return 8 * (-(-10 * n // 8) + 2)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("where", ["rhs", "matrix"])
@pytest.mark.parametrize("kind", ["tet", "cylinder"])
def test_nan_ends_as_at_the_limit(kind, where, mixed):
    m, J, P, b = setup(kind)
    for prec in (P, None):
        for max_iter in (1, 20, None):
            want = default_limit(m.ndof()) if max_iter is None else max_iter
            Jn, bn = J.clone(), b.clone()
            if where == "rhs":
                bn[m.ndof() // 2] = float("nan")
            else:
                Jn[m.nnz // 2] = float("nan")
            for engine in ("chunked", "streamed"):
                m.set_cg_engine(engine)
                x, k, it = solve(m, Jn, prec, bn, mixed, max_iter)
                assert k == H.SolveErrorKind.MaxIterationsReached and it == want
                assert torch.isnan(x).all()


@pytest.mark.parametrize("kind", ["tet", "cylinder"])
def test_nan_ends_as_in_the_graphs(kind):
    m, J, P, b = setup(kind)
    b[1] = float("nan")
    m.set_cg_engine("chunked")
    x, k, it = solve(m, J, P, b, False, None)
    m.set_spmv_variant(32)  # the graphs
    xg, kg, ig = solve(m, J, P, b, False, None)
    assert k == kg == H.SolveErrorKind.MaxIterationsReached and it == ig == default_limit(m.ndof())
    assert torch.isnan(x).all() and torch.isnan(xg).all()


@pytest.mark.parametrize("max_iter", [200, None])
@pytest.mark.parametrize("engine", ["chunked", "streamed"])
@pytest.mark.parametrize("kind", ["tet", "cylinder"])
def test_unreachable_tolerance_in_mixed_precision(kind, engine, max_iter):
    m, J, P, b = setup(kind)
    m.set_cg_engine(engine)
    x, k, it = solve(m, J, P, b, True, max_iter, tol=1e-17)
    assert it <= (default_limit(m.ndof()) if max_iter is None else max_iter)
    y = torch.zeros_like(b)
    m.spmv(y, J, x)
    # (200 iterations need not be enough for the cylinder)
    assert float((y - b).norm() / b.norm()) < (1e-10 if max_iter is None else 1.0)
