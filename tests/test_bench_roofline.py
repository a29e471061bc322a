"""The bench names a CG kernel, and counts its bytes, by what ran."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import bench


def variant(launches, engine):
    return {"cg_iterations": 700, "gpu_launches": launches, "phase_ms": {"cg": 35.0}, "cg_engine": engine}


def test_engine_on_the_csr_values():
    # 3 x 3 blocks of 1,000 node pairs, 100 nodes, subdomains of 27 and 8 nodes
    b = bench.csr_bytes_per_iteration(9000, 100, [27, 8], 8)
    assert b == 8 * 9000 + 4 * 1000 + 4 * 101 + 8 * (81 ** 2 + 24 ** 2) + 8 * 35
    csr = {"plain": b, "mixed": bench.csr_bytes_per_iteration(9000, 100, [27, 8], 4)}
    eng = {"auto_choice": 0, "launches": 0, "operator_bytes": 1, "schwarz_bytes": 1}  # (of the streamed layout)
    for head, key in (("plain", "plain"), ("mixed", "mixed"), ("learned", "mixed")):
        r = bench.cg_roofline(variant(20 * 350, eng), head, steps=20, csr_bytes=csr)
        assert r["kernel"].startswith("k_pcg") and r["bytes_per_iteration"] == csr[key]
        assert abs(r["achieved"] - csr[key] / 50e-6 / 1e9) < 1e-9 * r["achieved"]
        # four launches per iteration: the graphs
        r = bench.cg_roofline(variant(20 * 3000, eng), head, steps=20, csr_bytes=csr)
        assert "k_pcg" not in r["kernel"]


def test_streamed_engine():
    eng = {"auto_choice": 1, "launches": 5, "iterations": 700, "device_ms": 35.0, "operator_bytes": 10 ** 8,
           "schwarz_bytes": 10 ** 7}
    r = bench.cg_roofline(variant(100, eng), "mixed", steps=20, csr_bytes={"plain": 2, "mixed": 1})
    assert r["kernel"].startswith("k_cg_stream<float,float,2>") and r["bytes_per_iteration"] == 110000000
    assert bench.cg_roofline(variant(100, {}), "plain", steps=20) is None
