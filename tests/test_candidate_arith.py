"""Arithmetic of the candidate stage that stands in for the reference's form of
it (cctag_b200/csrc/cand_shared.hpp), on the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_convexity_intervals(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = tmp_path / "convexity"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "cctag_b200" / "csrc"),
                    "-I", str(ROOT / "include"), str(ROOT / "tests" / "cpp" / "convexity_test.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
