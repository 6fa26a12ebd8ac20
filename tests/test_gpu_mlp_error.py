"""Training after a tensor-core wait that ran out (tests/cpp/mlp_error_check.cu:
the error word is set by hand): the call reports it and leaves the weights and
the optimiser's moments as they were."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

pytestmark = pytest.mark.gpu


def test_weights_survive_a_failed_wait(tmp_path, torch_cuda):
    from finitevolumesolver_gb300 import build
    exe = tmp_path / "mlp_error_check"
    r = subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O2", "-I", str(ROOT / "include"),
                        "-I", str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "mlp_error_check.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "bad 0" in r.stdout, r.stdout + r.stderr
