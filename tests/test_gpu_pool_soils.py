"""Pools whose scenarios differ in soil, which take the update kernels that read
each scenario's own constants, and pools whose common soil changes while they
run, whose captured launches hold the constants: every scenario's results are
those of the same scenario alone, bit for bit (FP64: through swehr_advance, mixed:
alone in a pool), in both tile shapes (the tuner steps in both)."""
import numpy as np
import pytest

from swehr_b200 import workloads as W
from swehr_b200.params import FP64, MIXED

pytestmark = pytest.mark.gpu

SOILS = [
    dict(),
    dict(cohesion=5.0, J=12.0),
    dict(h0=0.0021, mtstar0=1.5, hf=0.07),
    dict(rhos=2400.0, phi=0.45, a=350.0, ad=900.0, uc=0.05, uc2=0.1),
    dict(g=9.7, hfilm=2e-5, thetas=0.45, theta0=0.12, F=0.03, betabedload=0.3, cthreshold=0.3),
]


def _case(soil, S, seed):
    return W.tiny_case(nx=20 + 3 * seed, ny=75 - 4 * seed, S=S, seed=seed, rain_mmh=300.0, tend=60.0 + 7.0 * seed,
                       **SOILS[soil])


def _alone(case, precision, max_steps=-1):
    from swehr_b200.lib import Pool, Simulation
    if precision == FP64:
        with Simulation(case) as s:
            pr = s.advance(max_steps=max_steps)
            return pr.steps, s.fields(), s.series()
    with Pool(precision=precision, max_classes=16) as pool:
        sc = pool.submit(case, max_steps=max_steps)
        pool.run(-1)
        return sc.progress().steps, sc.fields(), sc.series()


def _check(sc, case, precision, max_steps=-1):
    steps, fields, series = _alone(case, precision, max_steps)
    assert sc.progress().steps == steps
    got = sc.fields()
    for n in fields:
        assert np.array_equal(got[n], fields[n], equal_nan=True), n
    for a, b in zip(sc.series(), series):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("tune", [False, True], ids=["", "tuned"])
@pytest.mark.parametrize("counts", [(7, 7, 7), (10, 10, 10), (3, 2, 4), (8, 5, 7), (16, 1, 11)], ids=str)
def test_scenarios_of_different_soils(counts, tune, precision):
    from swehr_b200.lib import Pool
    cases = [_case(k % len(SOILS), S, k) for k, S in enumerate(counts + counts[:2])]
    with Pool(precision=precision, max_classes=max(8, max(counts))) as pool:
        scs = [pool.submit(c) for c in cases]
        if tune:
            pool.tune(4)
        pool.run(-1)
        for sc, c in zip(scs, cases):
            _check(sc, c, precision)


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("S", [4, 7])
def test_the_common_soil_changes_while_a_pool_runs(S, precision):
    """soil 1 alone, 1 and 3 together, 3 alone, 1 again, then 4: the launch
    shapes stay the same (equal grids and class counts), the constants do not."""
    from swehr_b200.lib import Pool

    def case(soil, seed):
        c = _case(soil, S, 3)
        c.topo = c.topo + 0.002 * np.random.default_rng(seed).standard_normal(c.topo.shape)
        return c

    with Pool(precision=precision, max_classes=16) as pool:
        live = []

        def submit(soil, seed, steps):
            c = case(soil, seed)
            live.append((pool.submit(c, max_steps=steps), c, steps))

        submit(1, 1, 60)
        pool.run(40)
        submit(3, 2, 70)
        pool.run(30)                 # the first ends inside
        pool.run(-1)
        for soil, seed in ((1, 3), (4, 4), (1, 5)):
            submit(soil, seed, 45)
            pool.run(-1)
        assert len(live) == 5
        for sc, c, steps in live:
            assert sc.progress().steps == steps
            _check(sc, c, precision, steps)
