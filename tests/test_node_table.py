"""The precompute's table of shared nodes (csrc/pc_nodes.cuh): claim, publication and the
order of the reads behind it, on the host (tests/cpp/node_table.cu; CPU, needs nvcc).
Results on a device do not show a read that is not ordered."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "g3lhalo_gb300", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not on PATH")
def test_nodes_are_read_behind_their_publication(tmp_path):
    exe = str(tmp_path / "node_table")
    r = subprocess.run(["nvcc", "-std=c++17", "-I", CSRC, "-o", exe, os.path.join(HERE, "cpp", "node_table.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
