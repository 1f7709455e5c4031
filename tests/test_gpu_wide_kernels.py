"""Runs whose constants are out of the ordinary kernels' range take kernels of
their own: in FP64 the plain operators (bit for bit the ordinary results, and the
oracle's), in the mixed form divisions by subnormal numbers, as without a film,
where a front's depths fall below the smallest normal FP32 number."""
import numpy as np
import pytest

from harness import OracleRun, compare, STATE_FIELDS, CLASS_FIELDS
from swehr_b200 import workloads as W
from swehr_b200.params import FP64, MIXED

pytestmark = pytest.mark.gpu

# constants that enter no result: the stream-power terms, where no flow exceeds the critical power
NO_POWER = dict(uc=1e300, uc2=1e300)
OUT = dict(NO_POWER, J=2.0 ** 101)
FLAT = dict(inflow=0, bndry=(1, 1, 1, 1), ks=0.0, per_cell_ks=False)


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
@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_results_are_the_ordinary_kernels(precision, S, budget):
    """Mixed: the compiler may fuse other multiply-adds (FP32 units in the last
    place, amplified over 150 steps)."""
    a, b = _fields(_case(S, **NO_POWER), precision, budget=budget), _fields(_case(S, **OUT), precision, budget=budget)
    if precision == FP64:
        assert a[0] == b[0] and a[2][0] == b[2][0]
    for n in a[1]:
        if precision == FP64:
            assert np.array_equal(a[1][n], b[1][n], equal_nan=True), n
        else:
            d = np.linalg.norm(a[1][n] - b[1][n])
            assert d <= 2e-5 * np.linalg.norm(a[1][n]), (n, d)


def test_fp64_equals_the_oracle():
    case = _case(5, rhos=2.0 ** 51, phi=1.0 - 2.0 ** -40)
    o = OracleRun(case, "shim")
    o.advance(max_steps=60)
    got = _fields(case, FP64, steps=60)[1]
    want = o.fields()
    res = compare(got, want, STATE_FIELDS + CLASS_FIELDS)
    assert all(v[2] for v in res.values()), res


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_a_pool_with_such_a_scenario(precision):
    """... while it runs beside ordinary ones, and after it has gone."""
    from swehr_b200.lib import Pool
    ordinary, odd = _case(5, nx=30), _case(7, nx=40, hfilm=0.0, **OUT)

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
            if precision == FP64:
                assert np.array_equal(g[f], want[f], equal_nan=True), f
            else:
                assert np.isfinite(g[f]).all(), f
                assert np.linalg.norm(g[f] - want[f]) <= 2e-5 * np.linalg.norm(want[f]), f


@pytest.mark.parametrize("timed", [False, True], ids=["", "timed"])
def test_mixed_without_a_film(timed):
    """Still depths down to 1e-19 m above a film of zero, whose 2.333rd power, the
    friction's divisor, is a subnormal FP32 number: as the FP64 form steps them,
    and no NaN (0 times an infinite reciprocal) among them."""
    from swehr_b200.lib import Simulation
    case = _case(3, nx=24, ny=64, hfilm=0.0, **dict(FLAT, ks=0.0))
    case.topo = np.zeros_like(case.topo)
    case.rain = np.zeros_like(case.rain)
    rng = np.random.default_rng(4)
    # flat patches of one depth each: their inner cells stay still
    h = np.repeat(np.repeat(10.0 ** rng.uniform(-19, -3, (3, 8)), 8, 0), 8, 1).astype(np.float32).astype(np.float64)
    out = []
    for precision in (FP64, MIXED):
        with Simulation(case, precision=precision) as s:
            s.set_timing(timed)
            s.write_field("h", h)
            s.advance(max_steps=1)
            out.append(s.fields())
    inner = np.zeros((24, 64), bool)
    for i in range(3):
        for j in range(8):
            inner[8 * i + 1: 8 * i + 7, 8 * j + 1: 8 * j + 7] = True
    for n in ("h", "hu", "hv", "maxvel", "z", "vinf", "totsed"):
        assert np.isfinite(out[1][n]).all(), n
        assert np.allclose(out[1][n][inner], out[0][n][inner], rtol=1e-6, atol=0), n


def test_mixed_velocities_below_1e_19():
    """Level water that hardly moves, on the ordinary kernels: its velocity's
    square is a subnormal FP32 number (1e-40 has 16 significant bits), whose root
    is the largest velocity.  Cells away from the walls."""
    from swehr_b200.lib import Simulation
    case = _case(2, nx=24, ny=64, **FLAT)
    case.topo = np.zeros_like(case.topo)
    case.rain = np.zeros_like(case.rain)
    out = []
    for precision in (FP64, MIXED):
        with Simulation(case, precision=precision) as s:
            s.write_field("h", np.full((24, 64), 1e-2))
            s.write_field("hu", np.full((24, 64), 1e-22))
            s.advance(max_steps=1)
            out.append(s.field("maxvel")[6:-6, 6:-6])
    assert (out[0] > 5e-21).all()
    assert np.abs(out[1] / out[0] - 1).max() < 1e-3


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


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
def test_slabs_of_such_a_run_equal_the_whole(precision):
    from swehr_b200.lib import Simulation, SlabDomain
    case = _case(4, nx=26, ny=40, hfilm=0.0, **OUT)
    names = ("h", "hu", "hv", "z", "vinf", "totsed", "U", "M")
    with Simulation(case, precision=precision) as s:
        pw = s.advance(max_steps=120)
        want = s.fields(names)
    with SlabDomain(case, 3, precision) as d:
        d.step(120)
        ps, got = d.progress(), d.fields(names)
    assert (ps.t, ps.dt, ps.steps) == (pw.t, pw.dt, 120)
    for n in names:
        assert np.array_equal(got[n], want[n], equal_nan=True), n
