"""Internal force kernels (csrc/forces.cu) against the FP64 oracle: 1e-10 of the
largest entry, the parity bound of the other FP64 assembly paths.  Element counts
around their CTAs (8 Tet10, 4 Hex27 elements), uniform and per-element rules of
one and several tiles of points (16 and 32), empty rules among them, distorted
elements, both materials, the staged and the colored launches, and collapsed
elements reported as singular.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TET, HEX = O.ELEM_TET10, O.ELEM_HEX27


def mesh(kind, elements, seed):
    s = (H.scenes.tet10_box if kind == TET else H.scenes.hex27_box)(1.0, 1, 1, 1, 3)
    conn = s.blocks[0].connectivity[:elements]
    used = np.unique(conn)
    X = s.vertices[used] + 0.02 * np.random.default_rng(seed).normal(size=(len(used), 3))
    return X, np.searchsorted(used, conn)


def rule(kind, points, rng):
    """Random points of the reference element (the kernels take any)."""
    p = rng.uniform(-1.0, 1.0, (points, 3))
    if kind == TET:
        l = rng.dirichlet([1.0] * 4, points)
        p = 2.0 * l[:, 1:] - 1.0
    return rng.uniform(0.5, 1.5, points) / max(points, 1), p


def models(kind, elements, points, seed):
    rng = np.random.default_rng(seed)
    X, conn = mesh(kind, elements, seed)
    ref = O.Scene(X)
    if np.isscalar(points):
        w, p = rule(kind, points, rng)
        m = H.NodalModel3d(X, conn, (w, p), kind)
        ref.add_block(kind, conn, w, p)
    else:  # a rule of its own per element, the last one uniform
        counts = rng.choice(points, elements)
        counts[:len(points)] = points[:elements]
        off = np.concatenate([[0], np.cumsum(counts)])
        w, p = rule(kind, int(off[-1]), rng)
        wu, pu = rule(kind, 9, rng)
        m = H.EmbeddedModel3d(X, conn[-1:], conn[:-1], (wu, pu), (off[:-1], w[:off[-2]], p[:off[-2]]), kind)
        ref.add_block(kind, conn[-1:], wu, pu)
        ref.add_block(kind, conn[:-1], w[:off[-2]], p[:off[-2]], off[:-1])
    ref.finalize_pattern()
    return m, ref


@pytest.mark.parametrize("material", [O.MAT_SNH, O.MAT_STVK])
@pytest.mark.parametrize("kind,elements,points", [
    (TET, 1, 14), (TET, 7, 1), (TET, 8, 4), (TET, 9, 16), (TET, 17, 17), (TET, 33, 40), (TET, 30, [0, 3, 16, 35]),
    (HEX, 1, 14), (HEX, 3, 1), (HEX, 4, 27), (HEX, 5, 32), (HEX, 9, 33), (HEX, 27, 70), (HEX, 21, [0, 2, 32, 65])])
def test_matches_oracle(kind, elements, points, material):
    m, ref = models(kind, elements, points, elements)
    mat = (H.StableNeoHookeanMaterial if material == O.MAT_SNH else H.StVKMaterial)(H.YoungPoisson(1e6, 0.4))
    ref.set_material(material, mat.lame.mu, mat.lame.lam, 1000.0)
    u = H.scenes.random_normal(elements, m.ndof(), 0.01)
    want = ref.forces(u)
    tol = 1e-10 * np.abs(want).max()
    for path in ("auto", "cuda_cores"):  # staged and colored
        m.set_stiffness_path(path)
        assert np.abs(m.assemble_elastic_pseudo_forces(u, mat) - want).max() <= tol, path
        assert np.abs(m.assemble_elastic_pseudo_forces_into_par(want.copy(), u, mat) - 2.0 * want).max() <= 2.0 * tol


@pytest.mark.parametrize("kind", [TET, HEX])
@pytest.mark.parametrize("cells", [2, 3, 5, 7])
def test_collapsed_elements_are_singular(kind, cells):
    s = (H.scenes.tet10_box if kind == TET else H.scenes.hex27_box)(1.0, 1, 1, 1, cells)
    b = s.blocks[0]
    m = H.NodalModel3d(s.vertices, b.connectivity, (b.weights, b.points), kind)
    mat = H.StableNeoHookeanMaterial(H.YoungPoisson(1e6, 0.4))
    flat = H.NodalModel3d(s.vertices * np.array([0.0, 1.0, 1.0]), b.connectivity, (b.weights, b.points), kind)
    for f in ("assemble_elastic_pseudo_forces", "assemble_stiffness"):
        with pytest.raises(H.HoefemError) as e:  # no volume in the reference state
            getattr(flat, f)(np.zeros(m.ndof()), mat)
        assert e.value.status == "SINGULAR"
        with pytest.raises(H.HoefemError) as e:  # F = 0 at every point, to rounding
            getattr(m, f)(-s.vertices.reshape(-1), mat)
        assert e.value.status == "SINGULAR"
        getattr(m, f)(np.zeros(m.ndof()), mat)  # the model stays usable
        # shrunk to a millionth: J = 1e-18, far above its rounding
        getattr(m, f)((1e-6 - 1.0) * s.vertices.reshape(-1), mat)
