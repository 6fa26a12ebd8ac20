"""AMR transfers while the default stream is busy.  The solver works on a stream
of its own that nothing orders behind the default stream, so a solver created,
filled, run and read while ordinary work of several lengths is queued there
gives the same bits as on an idle device."""
import numpy as np
import pytest

from finitevolumesolver_gb300 import workloads

pytestmark = pytest.mark.gpu

WORK = list(range(1, 13))  # passes over 1 GiB, a third of a millisecond each


def _busy(torch, n):
    x = torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    return lambda: [x.add_(1.0) for _ in range(n)]


@pytest.fixture(scope="module")
def problem(fvs):
    h, cons = workloads.amr_blast_2d(512, 3, target=1500)
    a = fvs.AmrSolver(h)
    a.upload(cons)
    a.run(cfl=0.8, t_end=10.0, max_steps=2)
    out = a.download()
    a.close()
    return h, cons, out


@pytest.mark.parametrize("work", WORK)
def test_first_upload(fvs, torch_cuda, problem, work):
    h, cons, ref = problem
    busy = _busy(torch_cuda, work)
    a = fvs.AmrSolver(h)
    busy()
    a.upload(cons)
    a.run(cfl=0.8, t_end=10.0, max_steps=2)
    np.testing.assert_array_equal(a.download(), ref)
    torch_cuda.cuda.synchronize()
    a.close()


@pytest.mark.parametrize("work", WORK)
def test_create(fvs, torch_cuda, problem, work):
    h, cons, ref = problem
    busy = _busy(torch_cuda, work)
    busy()
    a = fvs.AmrSolver(h)
    a.upload(cons)
    a.run(cfl=0.8, t_end=10.0, max_steps=2)
    np.testing.assert_array_equal(a.download(), ref)
    torch_cuda.cuda.synchronize()
    a.close()
