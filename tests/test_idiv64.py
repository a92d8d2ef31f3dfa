"""FP64 division on the integer pipes (csrc/idiv64.cuh) against the division operator.

Both are correctly rounded, so every quotient must agree in every bit (tolerance 0).
"""
import os
import subprocess

import pytest

from g3lhalo_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(tmp_path, *args):
    exe = str(tmp_path / "idiv64")
    subprocess.run([B.NVCC] + B.ARCH + ["-std=c++17", "-O3", "-fmad=false", "-Xcompiler",
                                        "-ffp-contract=off", "-I" + B.CSRC, "--expt-relaxed-constexpr",
                                        os.path.join(HERE, "cpp", "idiv64.cu"), "-o", exe], check=True)
    r = subprocess.run([exe] + list(args), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_host_quotients_match_bit_for_bit(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_device_quotients_match_bit_for_bit(tmp_path):
    _run(tmp_path, "gpu")
