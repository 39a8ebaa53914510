"""The pair terms' double root and quotient (mps_exact.cuh) where rounding is hardest: every root
within 2000 / 2^55 last places of the middle of two doubles, and quotients and reciprocals next to a
middle, of divisors at both ends of their binade and between. All must be the compiler's, bit for bit.
"""
from __future__ import annotations

import os
import subprocess

import pytest

from mps_cuda_b200.build import ARCH, nvcc_path

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_roots_and_quotients_next_to_a_middle(tmp_path):
    exe = str(tmp_path / "exact_hard")
    subprocess.run([nvcc_path(), *ARCH, "-O3", "-std=c++17", "-fmad=false",
                    os.path.join(HERE, "cpp", "exact_hard.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    *bad, n_root, n_quotient = [int(v) for v in out.split()]
    assert bad == [0, 0, 0, 0]  # roots, reciprocals, quotients, quotients by a given reciprocal
    assert n_root > 500 and n_quotient > 1_000_000
