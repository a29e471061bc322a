"""Schwarz blocks (csrc/precond.cu) whose nodes are stiff in one direction: every 3 x 3
pivot has one eigenvalue near 1 and two near 1 / kappa, as the nodes of slender cells
or of a nearly incompressible material have.

Reference: Gauss-Jordan elimination of the same stored blocks in extended precision
(64-bit significands, an error below 1e-11 at kappa = 1e8).  Elimination of a positive definite block of
dimension n in FP64 has a relative error of at most about n 2^-52 times its
condition: n <= 81 and a condition below 2 kappa here.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H

pytestmark = pytest.mark.gpu


def inverse(a):
    a = a.astype(np.longdouble)
    for k in range(len(a)):
        row, col = a[k].copy(), a[:, k].copy()
        piv = row[k]
        row[k], col[k] = 1, -1
        a[k], a[:, k] = 0, 0
        a -= np.outer(col, row / piv)
    return a


@pytest.mark.parametrize("nodes", [1, 10, 27])
@pytest.mark.parametrize("kappa", [1e2, 1e4, 1e6, 1e8])
def test_inverse_error_follows_the_condition(nodes, kappa):
    s = H.scenes.hex27_box(1.0, 1, 1, 1, 1)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points), b.kind)
    rng = np.random.default_rng(nodes)
    n = m.ndof()
    # symmetric couplings of up to 0.05 / n between unit directions, scaled by the
    # square root of every node's block
    E = rng.uniform(-0.05, 0.05, (n, n)) / n
    E = np.eye(n) + 0.5 * (E + E.T)
    root = np.zeros((n, n))
    for a in range(0, n, 3):
        Q = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        root[a:a + 3, a:a + 3] = (Q * np.sqrt([1.0, 1.3 / kappa, 1.0 / kappa])) @ Q.T
    A = root @ E @ root
    A = 0.5 * (A + A.T)
    sub = np.sort(rng.permutation(m.num_vertices)[:nodes])
    ro, ci = m.pattern()
    rows = np.repeat(np.arange(n), np.diff(ro))
    untreated = np.setdiff1d(np.arange(m.num_vertices), sub)
    P = H.SchwarzPreconditioner(m, [sub], untreated)
    P.update(A[rows, ci])
    d = (3 * sub[:, None] + np.arange(3)).reshape(-1)
    R = inverse(A[np.ix_(d, d)]).astype(np.float64)
    pro, pci = P.pattern()
    got = np.zeros((n, n))
    got[np.repeat(np.arange(n), np.diff(pro)), pci] = P.values()
    assert np.abs(got[np.ix_(d, d)] - R).max() <= 3 * nodes * 2.0 ** -52 * 2.0 * kappa * np.abs(R).max()
