"""Simulations and pools of different class counts share kernels, whose dynamic
shared memory limit is the process's: one made later for fewer classes leaves the
earlier one's launches possible.  The largest class count comes first here."""
import numpy as np
import pytest

from swehr_b200 import workloads as W
from swehr_b200.params import FP64, MIXED

pytestmark = pytest.mark.gpu


def _case(S, **kw):
    return W.tiny_case(nx=33, ny=40, S=S, seed=S, rain_mmh=300.0, tend=1e4, **kw)


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("budget", [False, True], ids=["", "budget"])
@pytest.mark.parametrize("counts", [(16, 11), (8, 5), (4, 2)])
def test_simulations(counts, budget, precision):
    from swehr_b200.lib import Simulation
    many, few = map(_case, counts)
    with Simulation(many, precision=precision, budget=budget) as a:
        a.advance(max_steps=70)
        want = a.fields()
    with Simulation(many, precision=precision, budget=budget) as a:
        with Simulation(few, precision=precision, budget=budget) as b:
            assert b.advance(max_steps=3).steps == 3
            assert a.advance(max_steps=70).steps == 70
            got = a.fields()
    for n in want:
        assert np.array_equal(want[n], got[n], equal_nan=True), n


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_pools(precision):
    from swehr_b200.lib import Pool, Simulation
    many, few = _case(16), _case(11)
    with Pool(precision=precision, max_classes=16) as a, Pool(precision=precision, max_classes=11) as b:
        sa, sb = a.submit(many), b.submit(few)
        b.run(3)
        a.run(40)
        got, steps = sa.fields(), sa.progress().steps
    assert steps == 40
    with Simulation(many, precision=precision) as s:
        s.advance(max_steps=steps)
        want = s.fields()
    if precision == FP64:
        for n in want:
            assert np.array_equal(want[n], got[n], equal_nan=True), n
    else:
        with Pool(precision=precision, max_classes=16) as a:
            sa = a.submit(many)
            a.run(40)
            want = sa.fields()
        for n in want:
            assert np.array_equal(want[n], got[n], equal_nan=True), n
