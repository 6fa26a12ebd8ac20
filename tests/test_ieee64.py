"""The integer-pipe quotients, square roots and comparisons of the FP64
flavours against the IEEE operations, bit for bit (tests/cpp/ieee64_check.cu):
the digit bounds on the host with perturbed seeds, and 2.7e8 operand pairs on
the device with the device's seeds."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def compile_check(tmp_path):
    from finitevolumesolver_gb300 import build
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = tmp_path / "ieee64_check"
    r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-O2", "-fmad=false",
                        "-I", str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "ieee64_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def test_host_digits(tmp_path):
    r = subprocess.run([str(compile_check(tmp_path))], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout + r.stderr


@pytest.mark.gpu
def test_device(tmp_path, torch_cuda):
    r = subprocess.run([str(compile_check(tmp_path)), "device"], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout + r.stderr
