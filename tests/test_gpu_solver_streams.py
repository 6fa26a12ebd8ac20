"""A uniform solver created, filled, run and read while ordinary work of several
lengths is queued on the default stream gives the same bits as on an idle
device: the solver works on a stream of its own that nothing orders behind the
default stream."""
import numpy as np
import pytest

from finitevolumesolver_gb300 import workloads

pytestmark = pytest.mark.gpu


def _run(fvs, cons, n):
    s = fvs.Solver([n, n], [1.0 / n] * 2, "periodic")
    s.upload(cons)
    st, dts = s.run(cfl=0.8, t_end=1e9, max_steps=40, log_len=40)
    out = s.download()
    s.close()
    return out, dts, st.steps


@pytest.mark.parametrize("work", [1, 2, 4, 6, 8, 12, 20, 40])
def test_create_and_run(fvs, torch_cuda, work):
    """`work` passes over 1 GiB, a third of a millisecond each; the 40 steps take
    about 5 ms."""
    n = 64
    cons = workloads.random_state((n, n), 2, seed=3, v=0.3).reshape(4, 1, n, n)
    ref = _run(fvs, cons, n)
    assert ref[2] == 40
    x = torch_cuda.zeros(1 << 28, device="cuda")
    torch_cuda.cuda.synchronize()
    for _ in range(work):
        x.add_(1.0)
    out = _run(fvs, cons, n)
    torch_cuda.cuda.synchronize()
    assert out[2] == 40
    np.testing.assert_array_equal(out[1], ref[1])
    np.testing.assert_array_equal(out[0], ref[0])
