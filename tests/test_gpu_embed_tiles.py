"""Candidate search of the embedding by tiles of 256 tets (csrc/embed.cu), and the
clip's early exits, against the oracle: tet counts around a tile and around the 256
tiles of a pass, spatially ordered and shuffled tets (tile boxes that meet every
cell).  Classes equal, cut volumes to 1e-13 of a cell, as the general test.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tets", [1, 255, 256, 257, 513, 1152])
@pytest.mark.parametrize("order", ["mesh", "shuffled", "behind"])
def test_candidates_of_every_tile(tets, order):
    bg = H.scenes.hex27_box(1.0, 1, 1, 1, 5)
    V, conn = bg.vertices, bg.blocks[0].connectivity
    X, T = H.scenes.hollow_cylinder_tets(0.3, 0.4, 1.0, 1, 24, 8)
    rng = np.random.default_rng(tets)
    assert len(T) >= tets
    T = (T if order == "mesh" else T[rng.permutation(len(T))])[:tets]
    if order == "behind":  # 257 tiles of tets that meet no cell come first
        far = len(X) + np.arange(4)
        X = np.concatenate([X, 50.0 + np.eye(4, 3)])
        T = np.concatenate([np.tile(far, (257 * 256 - tets // 2, 1)), T])
    emb, ref = H.embed_mesh_3d(V, conn, X, T), O.Embedding(V, conn, X, T)
    assert np.array_equal(emb.cell_class, ref.cell_class)
    assert np.abs(emb.cut_volume - ref.cut_volume).max() <= 1e-13 * 0.2 ** 3
    assert emb.cut_volume.max() > 0.0
