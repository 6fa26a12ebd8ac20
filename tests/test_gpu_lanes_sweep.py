"""One sweep with one cell per lane against one marching sweep on a weakly
disturbed state (1e-3), in the flavours whose two kernels may round differently:
a wrong neighbour, ghost or wall image moves a cell by 1e-4 or more.

The kernels take the same operations; only which products the compiler contracts
may differ, a rounding of the face flux each.  With dt/dx (|u| + c) <= 0.6 and
some ten roundings a face, two faces a cell, that is below 2 x 10 x 0.6 units of
the state's largest component: 2^-24 in mixed precision (7e-7), 2^-53 in fast FP64
(1.4e-15), 2^-44 for the double-float quotients and products (7e-13)."""
import numpy as np
import pytest

from finitevolumesolver_gb300 import workloads

pytestmark = pytest.mark.gpu

GRIDS = [(1,), (2,), (31,), (95,), (30, 3), (5, 31), (33, 34), (3, 4, 31), (32, 5, 2), (7, 30, 6)]
ROUNDING = {"mixed": 2.0 ** -24, "fp64_fast": 2.0 ** -53, "fp64_df": 2.0 ** -44}


@pytest.mark.parametrize("precision", list(ROUNDING))
@pytest.mark.parametrize("bc", ["periodic", "transmissive", "reflective"])
def test_one_sweep(fvs, bc, precision):
    for n in GRIDS:
        if bc == "reflective" and min(n) < 2:
            continue
        rank = len(n)
        rng = np.random.default_rng(sum(n))
        shape = tuple(reversed(n))
        one = lambda: 1.0 + 1e-3 * rng.standard_normal(shape)  # noqa: E731
        cons = workloads.cons_from_prim(one(), [0.2 * one() for _ in range(rank)], one())
        cons = cons.reshape((rank + 2,) + (1,) * (3 - rank) + shape)
        tol = 12 * ROUNDING[precision] * np.abs(cons).max()
        for d in range(rank):
            outs = []
            for seg in (1, 16):
                s = fvs.Solver(list(n), [1.0] * rank, bc,
                               method=fvs.make_method(precision=precision))
                variant = 10 if precision == "mixed" and d == 0 and seg != 1 else 0
                s.set_launch(d, seg, variant)
                s.upload(cons)
                s.sweep(d, 0.6 / 1.5)
                outs.append(s.download())
                s.close()
            assert np.abs(outs[0] - outs[1]).max() <= tol, (n, d)
