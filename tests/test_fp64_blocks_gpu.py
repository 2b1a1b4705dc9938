"""The FP64 lane's building blocks (rg_fp64.cuh) on the device, each against what it stands in for.

``tests/native/fp64_blocks_check.cu`` compares bits: quotients on random and on the hardest arguments,
the exponential and the logarithm, the exact forms, and the inverse normals of every 32-bit point.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

from riga_gb300.build import ARCH, nvcc

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def test_blocks_return_the_bits_they_stand_in_for(tmp_path):
    exe = tmp_path / "fp64_blocks_check"
    subprocess.run([nvcc(), *ARCH, "-std=c++17", "-O3", "-fmad=false", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "riga-flow_gb300" / "csrc"), str(ROOT / "tests" / "native" / "fp64_blocks_check.cu"),
                    "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
