"""Schwarz blocks (csrc/precond.cu) on ragged subdomains: node counts around the
inversion's tiles of three nodes (1, 2, 3, 4, 8, 9, 10, 17, 18, 19, 26, 27), an
indefinite block (the eigen path), and the apply from the blocks against the
apply of the assembled values.

Reference: numpy in FP64, the reference's spectrum rule (1 / |l|, floor
1e-12 max |l|).  The blocks are diagonally dominant (condition below 10), so the
rounding bound of either inverse is 81 * 2^-52 * 10, about 2e-13 relative: 1e-12.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H

pytestmark = pytest.mark.gpu


def setup(counts, seed, indefinite=()):
    s = H.scenes.hex27_box(1.0, 4, 2, 2, 1)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points), b.kind)
    rng = np.random.default_rng(seed)
    subs = [np.sort(rng.permutation(b.connectivity[k % len(b.connectivity)])[:n]) for k, n in enumerate(counts)]
    covered = np.zeros(m.num_vertices, dtype=bool)
    covered[np.concatenate(subs)] = True
    untreated = np.nonzero(~covered)[0]
    ro, ci = m.pattern()
    rows = np.repeat(np.arange(m.ndof()), np.diff(ro))
    A = np.zeros((m.ndof(), m.ndof()))
    A[rows, ci] = rng.normal(size=m.nnz)
    A = 0.5 * (A + A.T) / m.ndof()
    A[np.arange(m.ndof()), np.arange(m.ndof())] = 1.0 + rng.uniform(0.0, 1.0, m.ndof())
    for k in indefinite:
        d = 3 * subs[k][0]
        A[d, d] = -1.0
    return m, subs, untreated, A, A[rows, ci]


def reference(subs, untreated, A):
    P = np.zeros_like(A)
    for n in subs:
        d = (3 * n[:, None] + np.arange(3)).reshape(-1)
        l, V = np.linalg.eigh(A[np.ix_(d, d)])
        f = 1.0 / np.maximum(np.abs(l), 1e-12 * np.abs(l).max())
        P[np.ix_(d, d)] += (V * f) @ V.T
    d = (3 * untreated[:, None] + np.arange(3)).reshape(-1)
    P[d, d] = 1.0 / A[d, d]
    return P


@pytest.mark.parametrize("counts,indefinite", [([1, 2, 3], ()), ([4, 8, 9], ()), ([10, 17, 18, 3], ()), ([18, 2], (1,)),
                                               ([19, 26, 27, 1], ()), ([27] * 9, (4,)), ([27], ())])
def test_ragged_subdomains(counts, indefinite):
    m, subs, untreated, A, vals = setup(counts, len(counts), indefinite)
    P = H.SchwarzPreconditioner(m, subs, untreated)
    P.update(vals)
    R = reference(subs, untreated, A)
    r = np.random.default_rng(5).normal(size=m.ndof())
    z = P.apply(r)  # from the blocks
    assert np.abs(z - R @ r).max() <= 1e-12 * np.abs(R @ r).max()
    ro, ci = P.pattern()
    rows = np.repeat(np.arange(m.ndof()), np.diff(ro))
    assert np.abs(P.values() - R[rows, ci]).max() <= 1e-12 * np.abs(R).max()
    za = P.apply(r)  # now from the assembled values
    assert np.abs(za - z).max() <= 1e-12 * np.abs(z).max()
    P.update(vals)
    assert np.array_equal(P.apply(r), z)
