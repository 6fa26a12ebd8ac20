"""The nearly rounded quotients and square roots of the FP64 flavours against
their bounds of 0.57 and 0.75 units in the last place, and exact quotients
staying exact (tests/cpp/near64_check.cu): on the host with perturbed seeds, and
6.7e7 operand pairs on the device with the device's."""
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
    exe = tmp_path / "near64_check"
    r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-O2", "-fmad=false",
                        "-I", str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "near64_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout + r.stderr


def test_host(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_device(tmp_path, torch_cuda):
    _run(tmp_path, "device")
