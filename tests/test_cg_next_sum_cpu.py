"""The residual sums that the persistent CG forms ahead of the residual (host code,
csrc/cg_limit.h), compiled here with the host compiler (tests/cg_next_sum_test.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sums_that_are_taken_are_exact(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "cg_next_sum_test")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "higher_order_embedded_fem_b200", "csrc"),
                           "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cg_next_sum_test.cpp"),
                           "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
