"""What fvs_compute_stable_dt keeps between calls (a page-locked word and eight
bytes of the memory pool per thread): a thread that ends while another one
captures leaves the capture valid, and calls before and after cudaDeviceReset
return the same dt.  Each case is a process of its own."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

COMMON = """
import ctypes as C, sys, threading
sys.path.insert(0, {root!r})
import numpy as np
import finitevolumesolver_gb300 as fvs
from finitevolumesolver_gb300 import workloads
L = fvs.lib()
rt = C.CDLL("libcudart.so.13")
n = 64
cons = workloads.random_state((1, 1, n), 1, seed=2).reshape(3, n)
p = 0.4 * (cons[2] - 0.5 * cons[1] ** 2 / cons[0])
states = np.ascontiguousarray(np.concatenate([cons, [p], [np.sqrt(1.4 * p / cons[0])]]))
m = fvs.make_method()
box = fvs.box([0, 0, 0], [n, 1, 1])

def on_device():
    d = C.c_void_p()
    assert rt.cudaMalloc(C.byref(d), states.nbytes) == 0
    assert rt.cudaMemcpy(d, states.ctypes.data_as(C.c_void_p), states.nbytes, 1) == 0
    return d

def stable_dt(d):
    out = C.c_double(-1.0)
    r = L.fvs_compute_stable_dt(C.byref(m), 1, d, box, 1.0 / n, 0, 1, C.byref(out), None)
    assert r == 0, L.fvs_last_error()
    return out.value
"""

THREAD_END = """
d = on_device()
stream, graph, buf = C.c_void_p(), C.c_void_p(), C.c_void_p()
assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
assert rt.cudaMalloc(C.byref(buf), 256) == 0
called, end = threading.Event(), threading.Event()
def work():
    stable_dt(d)
    called.set()
    end.wait()
t = threading.Thread(target=work)
t.start()
called.wait()
assert rt.cudaStreamBeginCapture(stream, 0) == 0  # global: the strictest mode
end.set()
t.join()
assert rt.cudaMemsetAsync(buf, 0, 256, stream) == 0
assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0 and graph.value
print("ok", stable_dt(d))
"""

RESET = """
first = stable_dt(on_device())
called, end = threading.Event(), threading.Event()
def work():  # a thread whose word dies with the context before the thread ends
    assert stable_dt(on_device()) == first
    called.set()
    end.wait()
t = threading.Thread(target=work)
t.start()
called.wait()
for _ in range(3):
    assert rt.cudaDeviceReset() == 0
    d = on_device()
    assert stable_dt(d) == first and stable_dt(d) == first
end.set()
t.join()
assert stable_dt(d) == first
print("ok", first)
"""


@pytest.mark.parametrize("case", ["thread_end", "reset"])
def test_state(fvs, tmp_path, case):
    text = COMMON.format(root=str(ROOT)) + (THREAD_END if case == "thread_end" else RESET)
    r = subprocess.run([sys.executable, "-c", text], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
