"""FP64 Hex27 stiffness on the FP64 tensor cores (csrc/stiffness_hex27.cu)
against the FP64 oracle: 1e-10 of the largest entry, the parity bound of the other
FP64 assembly paths.  Uniform and per-element rules around its tiles (4 points in
the products, 32 in the point phase), empty rules among them, distorted elements,
both materials, and each output: staged blocks, colored scatter, dense element
matrices (under the projected stiffness).
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H
from oracle import oracle as O
from test_gpu_forces import models

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("material", [O.MAT_SNH, O.MAT_STVK])
@pytest.mark.parametrize("elements,points", [(1, 14), (3, 1), (2, 4), (5, 31), (9, 33), (27, 70), (21, [0, 2, 8, 27, 32, 65])])
def test_matches_oracle(elements, points, material):
    m, ref = models(O.ELEM_HEX27, elements, points, elements)
    mat = (H.StableNeoHookeanMaterial if material == O.MAT_SNH else H.StVKMaterial)(H.YoungPoisson(1e6, 0.4))
    ref.set_material(material, mat.lame.mu, mat.lame.lam, 1000.0)
    u = H.scenes.random_normal(elements, m.ndof(), 0.01)
    want = ref.stiffness(u)
    tol = 1e-10 * np.abs(want).max()
    for path in ("auto", "cuda_cores"):  # staged and colored
        m.set_stiffness_path(path)
        K = m.assemble_stiffness(u, mat)
        assert np.abs(K - want).max() <= tol, path
        assert np.abs(m.assemble_stiffness_into_par(want.copy(), u, mat) - 2.0 * want).max() <= 2.0 * tol
    projected = ref.stiffness_projected(u)
    K = m.assemble_projected_stiffness_into_par(np.zeros(m.nnz), u, mat)
    assert np.abs(K - projected).max() <= 1e-10 * np.abs(projected).max()
