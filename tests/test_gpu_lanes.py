"""The one-cell-per-lane sweep (segment length 1, the default on small grids)
against the marching sweep: line lengths around the 30 cells a warp owns, lines
of one and two cells, every boundary condition, flavour and flux family, grids
whose slot count ends inside a warp; and the patch fluxes with one cell per lane
against the oracle around the 31 faces a warp owns.

Exact units take the same operations in the same order: equal bits.  Where the
compiler may contract products (fast, double-float) the two kernels agree to the
flavours' 1e-12 per cell; mixed fluxes carry some ten FP32 roundings (1e-6
relative), which nine sweeps at a Courant number of 0.6 add up to 2e-5."""
import numpy as np
import pytest

from finitevolumesolver_gb300 import workloads
from tolerance import assert_close_fp64

pytestmark = pytest.mark.gpu

GRIDS = [(1,), (2,), (29,), (30,), (31,), (61,), (30, 3), (5, 31), (33, 32), (3, 4, 31),
         (32, 5, 2), (7, 30, 6)]
METHODS = [("muscl_hlle", "fp64_exact"), ("muscl_hlle", "fp64_fast"), ("muscl_hlle", "fp64_df"),
           ("muscl_hlle", "mixed"), ("hllem", "fp64_exact"), ("muscl_char", "fp64_exact"),
           ("godunov", "fp64_exact"), ("muscl_godunov", "fp64_exact")]


def _run(fvs, n, bc, flux, precision, cons, seg):
    m = fvs.make_method(flux, precision=precision,
                        guess="pvrs_tr" if "godunov" in flux else "mean")
    s = fvs.Solver(list(n), [1.0 / k for k in n], bc, method=m)
    for d in range(len(n)):
        s.set_launch(d, seg, 10 if precision == "mixed" and d == 0 and seg != 1 else 0)
    s.upload(cons)
    _, dts = s.run(cfl=0.6, t_end=1e9, max_steps=3, log_len=3)
    out = s.download()
    s.close()
    return out, dts


@pytest.mark.parametrize("flux,precision", METHODS)
@pytest.mark.parametrize("bc", ["periodic", "transmissive", "reflective"])
def test_lanes_match_marching(fvs, bc, flux, precision):
    for n in GRIDS:
        if bc == "reflective" and min(n) < 2:
            continue
        rank = len(n)
        cons = workloads.random_state(tuple(reversed(n)), rank, seed=sum(n), v=0.3)
        cons = cons.reshape((rank + 2,) + (1,) * (3 - rank) + tuple(reversed(n)))
        a, da = _run(fvs, n, bc, flux, precision, cons, 1)
        b, db = _run(fvs, n, bc, flux, precision, cons, 16)
        if precision == "fp64_exact":
            np.testing.assert_array_equal(da, db, err_msg=str(n))
            np.testing.assert_array_equal(a, b, err_msg=str(n))
        else:
            rtol = 2e-5 if precision == "mixed" else 1e-12
            np.testing.assert_allclose(da, db, rtol=10 * rtol, err_msg=str(n))
            assert_close_fp64(a, b, rank, rtol, str(n))


@pytest.mark.parametrize("kind", ["muscl_hlle", "muscl_hllem"])
@pytest.mark.parametrize("rank", [1, 2, 3])
def test_patch_fluxes_bit_exact(fvs, orc, torch_cuda, kind, rank):
    torch = torch_cuda
    okind = orc.MUSCL_HLLEM if kind == "muscl_hllem" else 0
    fm = fvs.FluxMethod(fvs.PerfectGas(rank), kind)
    for d in range(rank):
        for faces in (1, 30, 31, 32, 63):
            n = [3, 2, 3][:rank] + [1] * (3 - rank)
            n[d] = faces + 3  # cells of the faces' stencils
            lo = [-2, 1, -3]
            box_lo = [lo[k] if k < rank else 0 for k in range(3)]
            box_hi = [box_lo[k] + n[k] for k in range(3)]
            cons = workloads.random_state(tuple(reversed(n)), rank, seed=faces + rank)
            states = orc.complete_from_cons(rank, cons.reshape(rank + 2, -1))
            states = states.reshape((rank + 4,) + tuple(reversed(n)))
            flo, fhi = list(box_lo), list(box_hi)
            flo[d] += 2
            fhi[d] = flo[d] + faces
            shape = (rank + 2,) + tuple(fhi[k] - flo[k] for k in (2, 1, 0))
            out = torch.full(shape, float("nan"), dtype=torch.float64, device="cuda")
            st = torch.from_numpy(np.ascontiguousarray(states)).cuda()
            fm.ComputeNumericFluxes(out, (flo, fhi), st, (box_lo, box_hi), 1e-3, 0.05, d)
            torch.cuda.synchronize()
            ref = orc.compute_numeric_fluxes(orc.method(okind), rank, states, (box_lo, box_hi),
                                             (flo, fhi), 1e-3, 0.05, d)
            np.testing.assert_array_equal(out.cpu().numpy(), ref)
