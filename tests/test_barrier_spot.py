"""The FP64 lane's barrier thresholds against the rounded ratio itself, on the host.

The lane compares a spot with the smallest one whose ratio to its initial spot reaches the barrier;
this compiles ``tests/native/barrier_spot_check.cu`` against the engine library and tries both
neighbours of the threshold.  The search has to end for every pair that a request may hold: an absent
barrier (infinite) with an initial spot below 1 has its threshold far below infinity.  No GPU is used.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

from riga_gb300.build import build_library, nvcc

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "riga-flow_gb300" / "csrc"
LIBDIR = ROOT / "riga-flow_gb300" / "_build"


def test_thresholds_equal_the_rounded_ratio(tmp_path):
    build_library()
    exe = tmp_path / "barrier_spot_check"
    subprocess.run([nvcc(), "-std=c++17", "-O1", "-I", str(CSRC), str(ROOT / "tests" / "native" / "barrier_spot_check.cu"),
                    "-L", str(LIBDIR), "-lriga_gb300", "-Xlinker", f"-rpath={LIBDIR}", "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 wrong" in r.stdout
