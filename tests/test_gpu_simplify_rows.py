"""The quadrature simplification with a lane per moment (csrc/embed.cu,
k_simplify_rows: strengths 0 to 3): rules of 0 points up to several merge levels,
around its list sizes, random and tensor-grid points (ties in every pivot search),
zero weights and a degenerate (planar) rule.  The moments are kept to 1e-12 of the
largest, the tolerance of the general test, by a subset of at most r points in
order with positive weights; rules of at most r points stay as they are.
"""
import numpy as np
import pytest

import higher_order_embedded_fem_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strength,r", [(0, 1), (1, 4), (2, 10), (3, 20)])
@pytest.mark.parametrize("kind", ["random", "grid", "planar"])
def test_rules_of_every_size(strength, r, kind):
    rng = np.random.default_rng(10 * strength + len(kind))
    sizes = [0, 1, r - 1, r, r + 1, 2 * r - 1, 2 * r, 2 * r + 1, 4 * r, 4 * r + 1, 7 * r + 3, 17 * r, 900]
    rules = []
    for n in sizes:
        n = max(n, 0)
        if kind == "grid":
            g = np.linspace(-1.0, 1.0, 10)
            pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n]
        else:
            pts = rng.uniform(-1.0, 1.0, (n, 3))
            if kind == "planar":
                pts[:, 2] = 0.25
        w = rng.uniform(0.1, 1.0, n)
        if kind == "random" and n > 2 * r:
            w[rng.integers(0, n, n // 3)] = 0.0
        rules.append((w, pts))
    o = np.concatenate([[0], np.cumsum([len(w) for w, _ in rules])])
    w, p = np.concatenate([w for w, _ in rules]), np.concatenate([q for _, q in rules])
    oo, ow, op = H.embedding.simplify_rules(o, w, p, strength)
    for k, (wk, pk) in enumerate(rules):
        got_w, got_p = ow[oo[k]:oo[k + 1]], op[oo[k]:oo[k + 1]]
        if len(wk) <= r:
            assert np.array_equal(got_w, wk) and np.array_equal(got_p, pk)
            continue
        assert len(got_w) <= r and np.all(got_w > 0.0)
        idx = [int(np.nonzero((pk == q).all(1))[0][0]) for q in got_p]
        assert idx == sorted(set(idx))
        P = O.moment_matrix(pk, strength)
        m0 = P @ wk
        assert np.abs(P[:, idx] @ got_w - m0).max() <= 1e-12 * np.abs(m0).max()
