"""Comparisons that the selection settles from FP32 sums (csrc/sel_bound.cuh): each settled
one is the FP64 comparison, whatever the number of regions (tolerance 0).  On the host
(tests/cpp/sel_bound.cu; CPU, needs nvcc)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "g3lhalo_gb300", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_settled_comparisons_are_the_fp64_ones(tmp_path):
    exe = str(tmp_path / "sel_bound")
    r = subprocess.run(["nvcc", "-std=c++17", "-O3", "-Xcompiler", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                        os.path.join(HERE, "cpp", "sel_bound.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
