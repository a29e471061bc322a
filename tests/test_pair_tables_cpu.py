"""Node pair tables (host code, csrc/pair_tables.h), built by the compiler and
checked with the host compiler (tests/pair_tables_test.cpp)."""
import glob
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "higher_order_embedded_fem_b200", "csrc")


def test_tables_hold_their_identities(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "pair_tables_test")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "pair_tables_test.cpp"),
                           "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_no_table_is_copied_at_run_time():
    # a copy to a symbol goes through the default stream, after which a model's own
    # (non-blocking) stream does not wait
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        with open(path) as f:
            assert "cudaMemcpyToSymbol" not in f.read(), path
