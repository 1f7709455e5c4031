"""Domains stepped many steps a launch (k_run_tile) take the two kernels' steps
bit for bit: the per-launch timing path always runs two kernels a step, so the
same simulation advanced with and without it must end in the same state, time
and stage rows (and, where budgets keep it on two kernels, the same budgets).  Sizes around a tile (8 x 32), one block, every block
one tile, more tiles than blocks; steps around a launch's 128."""
import numpy as np
import pytest

from swehr_b200 import workloads as W
from swehr_b200.params import FP64, MIXED

pytestmark = pytest.mark.gpu

CASES = {
    "one_cell_wide": dict(nx=2, ny=2, S=1),
    "one_tile": dict(nx=8, ny=32, S=3),
    "tile_edges": dict(nx=9, ny=33, S=7, bndry=(1, 0, 0, 1)),
    "inflow": dict(nx=15, ny=51, S=4, inflow=1, bndry=(1, 0, 1, 1)),
    "two_tiles_a_block": dict(nx=180, ny=700, S=5),
    "ten_classes": dict(nx=70, ny=90, S=10),
    "sixteen_classes": dict(nx=33, ny=40, S=16),
}


def _result(s, case, stages):
    out = {n: a for n, a in s.fields().items()}
    if stages:
        out["stage"], out["saveflow"] = s.series()
    b = s.budget()
    out["budget"] = np.array([b.water_now, b.rain_in, b.outflow, b.clamp_gain, b.bulking, b.infiltration, b.rounding]
                             + [x for g in (b.sed_now, b.detach, b.sed_outflow, b.sed_rounding)
                                for x in g[:case.sclass]])
    return out


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("budget", [False, True], ids=["", "budget"])
@pytest.mark.parametrize("name", list(CASES))
def test_many_steps_a_launch_equal_two_kernels_a_step(name, budget, precision):
    from swehr_b200.lib import Simulation
    case = W.tiny_case(seed=3, rain_mmh=300.0, tend=1e4, **CASES[name])
    got = []
    for timed in (False, True):
        with Simulation(case, precision=precision, budget=budget) as s:
            s.set_timing(timed)
            steps = 0
            for n in (1, 127, 130):
                pr = s.advance(max_steps=n)
                steps += n
                assert pr.steps == steps and pr.status == 0
            s.set_timing(not timed)              # the other path goes on from this one's state
            pr = s.advance(max_steps=9)
            assert pr.steps == steps + 9
            got.append((pr.t, _result(s, case, True)))
    assert got[0][0] == got[1][0]
    for n in got[0][1]:
        assert np.array_equal(got[0][1][n], got[1][1][n], equal_nan=True), n


def test_a_run_ends_where_it_should():
    """t_stop, tend, the step limit and a CFL error inside a launch's steps."""
    from swehr_b200.lib import Simulation
    case = W.tiny_case(nx=20, ny=40, S=2, seed=4, rain_mmh=300.0, tend=20.0)
    ends = []
    for timed in (False, True):
        with Simulation(case) as s:
            s.set_timing(timed)
            a = s.advance(t_stop=3.3)
            b = s.advance(max_steps=5)
            c = s.advance()
            d = s.advance()
            assert c.done and d.steps_this_call == 0
            ends.append([(x.t, x.dt, x.courant, x.rain, x.steps, x.status) for x in (a, b, c, d)])
    assert ends[0] == ends[1]
    bad = W.tiny_case(nx=10, ny=10, S=2, seed=3, rain_mmh=500.0, tend=1000.0, cstable=40.0, maxstep=50.0)
    ends = []
    for timed in (False, True):
        with Simulation(bad) as s:
            s.set_timing(timed)
            a = s.advance()
            ends.append((a.t, a.steps, a.status, a.t_step, a.courant))
    assert ends[0] == ends[1] and ends[0][2] == 1
