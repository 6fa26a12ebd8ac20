"""Launch shapes of the FP64 AMR sweeps: the lanes of a warp along the rows (32
threads per row, the untuned shape) against the marching kernel in both
directions, with grids from one block (each warp loops over many slots) to more
than the level fills; and the shapes that the autotuner returns, which
set_launch takes.

Exact FP64 takes the same operations in the same order: equal bits.  Fast FP64
may contract products differently in the two kernels: the flavour's 1e-12 per
cell and sweep, over the 84 sweeps of three coarse steps on three levels."""
import numpy as np
import pytest

from finitevolumesolver_gb300 import workloads

pytestmark = pytest.mark.gpu

SHAPES = [(1, 128, 64), (8, 32, 2), (32, 32, 1), (32, 64, 3), (32, 128, 5000)]


def _run(fvs, h, cons, precision, shapes):
    a = fvs.AmrSolver(h, fvs.make_method(precision=precision))
    for (level, d), (tpr, block, grid) in shapes.items():
        a.set_launch(level, d, block, grid, tpr)
    a.upload(cons)
    st, dts = a.run(cfl=0.8, t_end=10.0, max_steps=3, log_len=3)
    assert st.steps == 3
    out = a.download()
    a.close()
    return out, dts


@pytest.mark.parametrize("bc", [(0, 0), (1, 1), (2, 2)])
@pytest.mark.parametrize("precision", ["fp64_exact", "fp64_fast"])
def test_lanes_match_marching(fvs, precision, bc):
    h, cons = workloads.amr_blast_2d(96, 3, target=150, sizes=(8, 16, 32))
    h = workloads.AmrHierarchy(h.nlevels, h.n0, bc, h.dx0, h.levels, h.boxes)
    ref, ref_dts = _run(fvs, h, cons, precision, {})
    for shape in SHAPES:
        for dirs in ((0,), (1,), (0, 1)):
            out, dts = _run(fvs, h, cons, precision,
                            {(l, d): shape for l in range(3) for d in dirs})
            if precision == "fp64_exact":
                np.testing.assert_array_equal(dts, ref_dts, err_msg=str(shape))
                np.testing.assert_array_equal(out, ref, err_msg=str(shape))
            else:
                np.testing.assert_allclose(dts, ref_dts, rtol=1e-10, err_msg=str(shape))
                np.testing.assert_allclose(out, ref, rtol=0, atol=84e-12 * np.abs(ref).max(),
                                           err_msg=str(shape))


@pytest.mark.parametrize("precision", ["fp64_exact", "fp64_fast", "mixed"])
def test_tuned_shapes_are_accepted(fvs, precision):
    h, cons = workloads.amr_blast_2d(96, 3, target=150, sizes=(8, 16, 32))
    a = fvs.AmrSolver(h, fvs.make_method(precision=precision))
    a.upload(cons)
    cfg = a.autotune()
    for level in range(3):
        for d in range(2):
            block, grid, tpr = (int(v) for v in cfg[level, d])
            a.set_launch(level, d, 64, 1, 1)
            a.set_launch(level, d, block, grid, tpr)
    a.close()
