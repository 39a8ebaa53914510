"""The pair terms' root and quotient (mps_exact.cuh) against the compiler's correctly rounded ones:
every single-precision significand, and 33 million random double operands, must agree bit for bit.
"""
from __future__ import annotations

import os
import subprocess

import pytest

from mps_cuda_b200.build import ARCH, nvcc_path

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_root_and_quotient_round_correctly(tmp_path):
    exe = str(tmp_path / "exact_arith")
    subprocess.run([nvcc_path(), *ARCH, "-O3", "-std=c++17", "-fmad=false",
                    os.path.join(HERE, "cpp", "exact_arith.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    assert [int(v) for v in out.split()] == [0] * 8
