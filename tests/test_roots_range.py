"""The exact Riemann solver's x^(-1/n) over the whole range of ratios that it
takes and for root orders from 3 to 64, against an extended-precision power,
within 2.9 units of 2^-53 (tests/cpp/root_device_check.cu): on the host, and on
the device, whose FP32 estimate of the root is another one."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def _run(tmp_path, *args):
    from finitevolumesolver_gb300 import build
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = tmp_path / "root_device_check"
    r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-O2", "-fmad=false",
                        "-I", str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "root_device_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "fail 0" in r.stdout, r.stdout + r.stderr


def test_host(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_device(tmp_path, torch_cuda):
    _run(tmp_path, "device")
