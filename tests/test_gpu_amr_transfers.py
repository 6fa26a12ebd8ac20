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


def _tiles(n, cells, bc=(0, 0)):
    boxes = [(x, y, min(x + cells, n), min(y + cells, n))
             for y in range(0, n, cells) for x in range(0, n, cells)]
    return workloads.AmrHierarchy(1, (n, n), bc, 1.0 / n, [0] * len(boxes), boxes)


@pytest.mark.parametrize("n,cells", [(1800, 1800), (1800, 600), (1800, 70), (1800, 60), (192, 24)])
def test_round_trip(fvs, n, cells):
    """Patches from one that fills the level (104 MB, more than the transfers'
    buffer) to ones that share a block's part: what was uploaded comes back, and
    one step of it matches the uniform grid's."""
    h = _tiles(n, cells)
    cons = workloads.random_state((n, n), 2, seed=n + cells)
    flat = np.concatenate([cons[:, y0:y1, x0:x1].reshape(-1) for (x0, y0, x1, y1) in h.boxes])
    a = fvs.AmrSolver(h)
    a.upload(flat)
    np.testing.assert_array_equal(a.download(), flat)
    a.run(cfl=0.5, t_end=10.0, max_steps=1)
    out = a.download()
    a.close()
    s = fvs.Solver([n, n], [1.0 / n] * 2, "periodic")
    s.upload(cons.reshape(4, 1, n, n))
    s.run(cfl=0.5, t_end=10.0, max_steps=1)
    ref = s.download().reshape(4, n, n)
    s.close()
    np.testing.assert_array_equal(
        out, np.concatenate([ref[:, y0:y1, x0:x1].reshape(-1) for (x0, y0, x1, y1) in h.boxes]))


def test_transfers_take_bounded_memory(fvs, torch_cuda):
    """Nothing of the size of the state is allocated by a transfer."""
    torch = torch_cuda
    n = 1800
    h = _tiles(n, n)
    a = fvs.AmrSolver(h)
    flat = np.ones(4 * n * n)
    free = torch.cuda.mem_get_info()[0]
    a.upload(flat)
    a.download()
    assert free - torch.cuda.mem_get_info()[0] <= 8 << 20
    a.close()
