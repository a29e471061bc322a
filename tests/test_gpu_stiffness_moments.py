"""FP64 Tet10 stiffness from moments of the tangent (csrc/stiffness_moments.cu)
against the FP64 oracle: 1e-10 of the largest entry, the parity bound of the
other FP64 assembly paths.  Sizes around its eight-element CTAs, every rule it
takes (1 to 14 points, and 20: two tiles of 16), distorted elements, both
materials, and a collapsed element reported as singular.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rule(points):
    if points in (1, 4, 6, 14):
        return H.tet_quadrature_strength({1: 1, 4: 2, 6: 3, 14: 5}[points])
    # the concatenation of two rules, each with half its weights: exact where both are
    (w1, p1), (w2, p2) = H.tet_quadrature_strength(3), H.tet_quadrature_strength(5)
    return np.concatenate([0.5 * w1, 0.5 * w2]), np.concatenate([p1, p2])


def model(elements, points, kind, seed):
    s = H.scenes.tet10_box(1.0, 1, 1, 1, 3)
    conn = s.blocks[0].connectivity[:elements]
    used = np.unique(conn)
    X = s.vertices[used] + 0.02 * np.random.default_rng(seed).normal(size=(len(used), 3))
    conn = np.searchsorted(used, conn)
    w, p = rule(points)
    m = H.NodalModel3d(X, conn, (w, p))
    mat = (H.StableNeoHookeanMaterial if kind == O.MAT_SNH else H.StVKMaterial)(H.YoungPoisson(1e6, 0.4))
    ref = O.Scene(X)
    ref.add_block(O.ELEM_TET10, conn, w, p)
    ref.finalize_pattern()
    ref.set_material(kind, mat.lame.mu, mat.lame.lam, 1000.0)
    return m, mat, ref, X, conn


@pytest.mark.parametrize("kind", [O.MAT_SNH, O.MAT_STVK])
@pytest.mark.parametrize("elements,points", [(1, 14), (7, 14), (8, 1), (9, 4), (17, 6), (162, 14), (33, 20)])
def test_matches_oracle(elements, points, kind):
    m, mat, ref, X, conn = model(elements, points, kind, elements)
    u = H.scenes.random_normal(elements, m.ndof(), 0.01)
    K, R = m.assemble_stiffness(u, mat), ref.stiffness(u)
    assert np.abs(K - R).max() <= 1e-10 * np.abs(R).max()
    # adds into the values
    K2 = m.assemble_stiffness_into_par(K.copy(), u, mat)
    assert np.abs(K2 - 2 * R).max() <= 2e-10 * np.abs(R).max()


def test_collapsed_elements_are_singular():
    s = H.scenes.tet10_box(1.0, 1, 1, 1, 3)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points))
    mat = H.StableNeoHookeanMaterial(H.YoungPoisson(1e6, 0.4))
    with pytest.raises(H.HoefemError) as e:
        m.assemble_stiffness(-s.vertices.reshape(-1), mat)  # F = 0 at every point
    assert e.value.status == "SINGULAR"
    m.assemble_stiffness(np.zeros(m.ndof()), mat)  # the model stays usable
