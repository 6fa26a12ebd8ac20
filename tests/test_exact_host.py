"""Pieces of the exact FP64 physics, compiled for the host, against the
reference's expressions in IEEE arithmetic, bit for bit
(tests/cpp/exact_host_check.cpp): signed zeros, ties, subnormals, infinities,
NaN and numbers of every exponent."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_exact_pieces(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = tmp_path / "exact_host_check"
    r = subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off",
                        "-I", str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "exact_host_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout + r.stderr
