"""Handles of different sizes launch the same kernels: a kernel's limit of dynamic
shared memory is the device's, so setting it up for a small handle must not
refuse the launches of a larger one, neither in turn on one host thread nor from
two threads with a model each.

Each launch is refused or runs whole, so results are compared bit by bit with those of
the handle alone.
"""
import threading

import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def schwarz(nodes):
    s = H.scenes.hex27_box(1.0, 4, 2, 2, 1)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points), b.kind)
    subs = [np.sort(c[:nodes]) for c in b.connectivity[:5]]
    covered = np.zeros(m.num_vertices, dtype=bool)
    covered[np.concatenate(subs)] = True
    ro, ci = m.pattern()
    rows = np.repeat(np.arange(m.ndof()), np.diff(ro))
    vals = np.random.default_rng(nodes).normal(size=m.nnz) / m.ndof()
    vals[rows == ci] = 1.5
    return m, H.SchwarzPreconditioner(m, subs, np.nonzero(~covered)[0]), vals


@pytest.mark.parametrize("order", [(27, 1), (27, 18, 9), (18, 2), (9, 27, 1)])
def test_preconditioners_of_different_sizes_in_turn(order):
    made = [schwarz(n) for n in order]
    r = np.random.default_rng(1).normal(size=made[0][0].ndof())
    z = []
    for k in range(2):
        for m, P, vals in made:
            P.update(vals)
            z.append(P.apply(r))
    n = len(made)
    for k in range(n):
        assert np.isfinite(z[k]).all() and np.array_equal(z[k], z[n + k])


def cg_problem(cells, quad):
    s = H.scenes.tet10_box(1.0 / cells, cells, cells, cells, quad)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points))
    mat = H.StableNeoHookeanMaterial(H.YoungPoisson(1e6, 0.4))
    u = np.zeros(m.ndof())
    J = torch.from_numpy(1e-6 * m.assemble_stiffness(u, mat) + m.assemble_mass(1000.0)).cuda()
    m.set_cg_engine("chunked")
    P = H.DiagonalPreconditioner(m)
    P.update(J)
    return m, J, P, torch.from_numpy(H.scenes.random_normal(4, m.ndof(), 1.0)).cuda()


def solve(p):
    m, J, P, b = p
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    (H.ConjugateGradient(m).with_operator(J).with_preconditioner(P)
     .with_stopping_criterion(H.RelativeResidualCriterion(1e-8)).solve_with_guess(b, x))
    return x


def run_threads(jobs, repeats):
    errors = []

    def work(fn, want):
        try:
            for _ in range(repeats):
                if not fn(want):
                    raise AssertionError("another result")
        except Exception as e:  # (a thread's exception would be lost)
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_solves_of_two_threads():
    problems = [cg_problem(1, 1), cg_problem(9, 1)]
    run_threads([(lambda want, p=p: torch.equal(solve(p), want), solve(p)) for p in problems], 200)


def test_preconditioner_updates_of_two_threads():
    jobs = []
    for nodes in (20, 27):
        m, P, vals = schwarz(nodes)
        r = np.ones(m.ndof())

        def once(want, P=P, vals=vals, r=r):
            P.update(vals)
            return np.array_equal(P.apply(r), want)

        P.update(vals)
        jobs.append((once, P.apply(r)))
    run_threads(jobs, 200)
