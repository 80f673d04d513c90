"""The rule for the blocks and warps of an identification launch, on the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_ident_layout(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = tmp_path / "ident_layout"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "cctag_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "ident_layout_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
