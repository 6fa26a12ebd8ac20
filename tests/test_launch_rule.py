"""The automatic segment length of the uniform sweeps (csrc/fvs_launch_rule.h):
on the host over sizes up to the largest that a direction takes, and on the
device for long, narrow mixed grids."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def auto(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = tmp_path_factory.mktemp("rule") / "launch_rule"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I",
                    str(ROOT / "finitevolumesolver_gb300" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "launch_rule.cpp"), "-o", str(exe)], check=True)

    def run(cases):
        text = "".join(" ".join(f"{k}={int(v)}" for k, v in c.items()) + "\n" for c in cases)
        r = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True)
        return [int(v) for v in r.stdout.split()]

    return run


def _segments(n, seg):
    return -(-n // seg)


LENGTHS = sorted({m for k in range(31) for m in ((1 << k) - 1, 1 << k, (1 << k) + 1)
                  if 0 < m < 1 << 31} | {100000, 524280, 524281, 524289, 600000, 1000000, 1048561})


def test_segments_fit_a_launch(auto):
    """A marching sweep's segments of a line are the grid's second dimension, at
    most 65535; one cell per lane counts its slots in 32 bits."""
    cases = [dict(rank=rank, cells=n * other, n=n, mixed=mixed, cut_cells=cc, family=family)
             for n in LENGTHS for other in (1, 2, 4, 1000, 1 << 20)
             for rank in (1, 2, 3) for mixed in (0, 1) for cc in (0, 1) for family in range(3)
             if (rank > 1 or other == 1) and (rank == 2 or not cc) and n * other < 1 << 34]
    for c, seg in zip(cases, auto(cases)):
        assert 1 <= seg <= max(c["n"], 1), c
        if seg == 1 and not c["cut_cells"] and c["n"] > 1:
            assert c["cells"] // c["n"] * (c["n"] + 2) < 1 << 31, c
        else:
            assert _segments(c["n"], seg) <= 65535, c


@pytest.mark.parametrize("mixed,variants", [(0, (3,)), (1, (4, 5, 10, 14, 15, 20, 24, 25))])
def test_a_chosen_variant_marches(auto, mixed, variants):
    """fvs_solver_set_launch(dir, 0, variant): the automatic length of that
    variant of the marching sweep, never one cell per lane."""
    cases = [dict(rank=rank, cells=n ** rank, n=n, mixed=mixed, variant=v)
             for rank in (1, 2, 3) for n in (16, 25, 64, 160) for v in (0, *variants)]
    for c, seg in zip(cases, auto(cases)):
        if c["variant"]:
            assert seg > 1, c
        elif not mixed:
            assert seg == 1, c


# (family, n of the direction, other extents' product, rank): one cell per lane?
# (HLLE: fast FP64 and double-float, then exact)
HLLE, HLLEM, GODUNOV = range(3)
MEASURED = [(HLLE, 160, 160 ** 2, 3, True), (HLLE, 192, 192 ** 2, 3, False),
            (HLLE, 1600, 1600, 2, True), (HLLE, 1800, 1800, 2, False),
            (HLLE, 1 << 22, 1, 1, True), (HLLEM, 2048, 2048, 2, True),
            (HLLEM, 160, 160 ** 2, 3, True), (GODUNOV, 80, 80 ** 2, 3, True),
            (GODUNOV, 96, 96 ** 2, 3, False), (GODUNOV, 128, 128 ** 2, 3, False),
            (GODUNOV, 512, 512, 2, True), (GODUNOV, 512, 1024, 2, True),
            (GODUNOV, 2048, 2048, 2, True), (GODUNOV, 64, 8192, 2, False),
            (GODUNOV, 8192, 64, 2, True), (GODUNOV, 64, 2048, 2, True),
            (GODUNOV, 1 << 22, 1, 1, True)]


def test_one_cell_per_lane_where_it_is_faster(auto):
    """The side of the rule that each measured sweep falls on."""
    cases = [dict(family=f, n=n, cells=n * other, rank=rank) for f, n, other, rank, _ in MEASURED]
    for m, seg in zip(MEASURED, auto(cases)):
        assert (seg == 1) == m[4], m
    exact = [dict(family=HLLE, n=n, cells=n ** 2, rank=2, exact=1) for n in (1800, 2048, 2100)]
    assert [seg == 1 for seg in auto(exact)] == [True, True, False]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(2, 600000), (2, 2, 600000)])
def test_long_narrow_mixed_grid(fvs, n):
    from finitevolumesolver_gb300 import workloads
    rank = len(n)
    cons = workloads.random_state(tuple(reversed(n)), rank, seed=1, v=0.3)
    cons = cons.reshape((rank + 2,) + (1,) * (3 - rank) + tuple(reversed(n)))
    outs = []
    for seg in (0, 16):
        s = fvs.Solver(list(n), [1.0] * rank, "periodic", method=fvs.make_method(precision="mixed"))
        if seg:
            s.set_tiling(seg)
        s.upload(cons)
        s.run(cfl=0.5, t_end=1e9, max_steps=1)
        outs.append(s.download())
        s.close()
    np.testing.assert_array_equal(outs[0], outs[1])
