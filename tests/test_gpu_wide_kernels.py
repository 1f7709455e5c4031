"""Runs whose constants are out of the ordinary kernels' range take kernels of
their own, in FP64 the plain operators: bit for bit the ordinary results, and the
oracle's."""
import numpy as np
import pytest

from harness import OracleRun, compare, STATE_FIELDS, CLASS_FIELDS
from swehr_b200 import workloads as W
from swehr_b200.params import FP64

pytestmark = pytest.mark.gpu

# constants that enter no result: the stream-power terms, where no flow exceeds the critical power
NO_POWER = dict(uc=1e300, uc2=1e300)
OUT = dict(NO_POWER, J=2.0 ** 101)


def _case(S=4, nx=21, ny=70, **over):
    return W.tiny_case(nx=nx, ny=ny, S=S, seed=8, rain_mmh=300.0, tend=1e4, **over)


def _fields(case, precision, steps=150, budget=False, timed=False):
    from swehr_b200.lib import Simulation
    with Simulation(case, precision=precision, budget=budget) as s:
        s.set_timing(timed)
        pr = s.advance(max_steps=steps)
        b = s.budget()
        return pr.t, s.fields(), [b.water_now, b.outflow, b.bulking]


@pytest.mark.parametrize("budget", [False, True], ids=["", "budget"])
@pytest.mark.parametrize("S", [1, 7, 16])
@pytest.mark.parametrize("precision", [FP64], ids=["fp64"])
def test_results_are_the_ordinary_kernels(precision, S, budget):
    a, b = _fields(_case(S, **NO_POWER), precision, budget=budget), _fields(_case(S, **OUT), precision, budget=budget)
    assert a[0] == b[0] and a[2][0] == b[2][0]
    for n in a[1]:
        assert np.array_equal(a[1][n], b[1][n], equal_nan=True), n


def test_fp64_equals_the_oracle():
    case = _case(5, rhos=2.0 ** 51, phi=1.0 - 2.0 ** -40)
    o = OracleRun(case, "shim")
    o.advance(max_steps=60)
    got = _fields(case, FP64, steps=60)[1]
    want = o.fields()
    res = compare(got, want, STATE_FIELDS + CLASS_FIELDS)
    assert all(v[2] for v in res.values()), res


@pytest.mark.parametrize("precision", [FP64], ids=["fp64"])
def test_a_pool_with_such_a_scenario(precision):
    """... while it runs beside ordinary ones, and after it has gone."""
    from swehr_b200.lib import Pool
    ordinary, odd = _case(5, nx=30), _case(7, nx=40, **OUT)

    def alone(c, steps):
        with Pool(precision=precision, max_classes=8) as p:
            sc = p.submit(c, max_steps=steps)
            p.run(-1)
            return sc.fields()

    with Pool(precision=precision, max_classes=8) as p:
        a, b = p.submit(ordinary, max_steps=90), p.submit(odd, max_steps=50)
        p.tune(2)
        p.run(-1)
        got = [a.fields(), b.fields()]
        assert (a.progress().steps, b.progress().steps) == (90, 50)
    for g, c, n in zip(got, (ordinary, odd), (90, 50)):
        want = alone(c, n)
        for f in want:
            assert np.array_equal(g[f], want[f], equal_nan=True), f


def test_such_a_run_forms_each_cell_once():
    """FP64, 200 x 50 hillslope in ponded flow: 1.55 times the ordinary kernels'
    step with the plain operators, 2.5 with both."""
    from swehr_b200.lib import Simulation
    us = []
    for over in (NO_POWER, OUT):
        c = W.hillslope200x50()
        c.params.update(over)
        with Simulation(c) as s:
            s.advance(max_steps=1500)
            pr = s.advance(max_steps=700)
            us.append(pr.device_ms / pr.steps_this_call)
    assert us[1] < 2.0 * us[0], us
