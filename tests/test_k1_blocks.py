"""K1's cut of a case's radii into blocks (lmie_b200/csrc/k1_blocks.h) on the
CPU: a block's radii fit its shared memory whatever their order."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_blocks_fit_their_rows_for_radii_in_any_order(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "k1_blocks_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", str(ROOT / "lmie_b200" / "csrc"),
                    str(ROOT / "tests" / "k1_blocks_check.cc"), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr
