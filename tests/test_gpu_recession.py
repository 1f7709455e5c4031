"""Suspended mass that has settled by hundreds of powers of ten, as after the
rain: U_k from 2^-780 down through the subnormals, where a decay by less than a
half rounds to none and a few units stay as long as the water flows.  The cells
that hold it give the plain operators' results and are not computed twice.

The plain operators are reached by a constant outside the sequences' range that
enters no result (F = 2^101 with critical powers that no flow exceeds)."""
import numpy as np
import pytest

from swehr_b200 import workloads as W

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -1074


def _case(S, F):
    c = W.tiny_case(nx=21, ny=43, S=S, seed=8, rain_mmh=300.0, tend=1e4, F=F, uc=1e300, uc2=1e300)
    c.rain = np.array([300.0, 0.0, 0.0]) * W.MMH
    c.params["rint"] = 3.0
    return c


def _settled(S, kind, rng, shape):
    """U_k of every class"""
    if kind == "decaying":                               # all of them, through the bound and the subnormals
        return [rng.uniform(1, 2, shape) * 2.0 ** rng.integers(-1040, -780, shape) for _ in range(S)]
    if kind == "stuck":
        return [UNIT * rng.integers(0, 4, shape) for _ in range(S)]
    if kind == "beside_large":                           # the first class is what the others are lost in
        return [rng.uniform(1e-9, 1e-6, shape) if k == 0 else UNIT * rng.integers(0, 2 ** 40, shape) for k in range(S)]
    out = []                                             # mixed: every size, signs too
    for _ in range(S):
        u = rng.uniform(-1, 2, shape) * 2.0 ** rng.choice([-1070, -1000, -861, -859, -830, -796, -700, -20], shape)
        out.append(np.where(rng.random(shape) < 0.3, 0.0, u))
    return out


def _run(c, kind, budget, timed):
    from swehr_b200.lib import Simulation
    rng = np.random.default_rng(2)
    out = []
    with Simulation(c, budget=budget) as s:
        s.set_timing(timed)
        s.advance(t_stop=4.0)
        for n in ("h", "hu", "hv"):
            s.write_field(n, {"h": 4e-3, "hu": 1e-4, "hv": -5e-5}[n] * rng.uniform(0.5, 1.5, (c.nx, c.ny)))
        s.write_field("h", np.where(rng.random((c.nx, c.ny)) < 0.1, 9e-5, s.field("h")))
        for k, u in enumerate(_settled(c.sclass, kind, rng, (c.nx, c.ny))):
            s.write_field("U", u, k + 1)
        for n in (1, 1, 1, 7, 40):
            pr = s.advance(max_steps=n)
            b = s.budget()
            out.append((pr.t, pr.dt, s.fields(), [b.water_now, b.outflow, b.bulking, b.rounding] + list(b.sed_outflow)))
    return out


@pytest.mark.parametrize("budget", [False, True], ids=["", "budget"])
@pytest.mark.parametrize("kind", ["decaying", "stuck", "beside_large", "mixed"])
@pytest.mark.parametrize("S", [1, 7, 12])
def test_settled_states_equal_the_plain_operators(S, kind, budget):
    plain = _run(_case(S, 2.0 ** 101), kind, budget, True)
    if kind == "stuck":
        assert all((f["U"] > 0).any() for _, _, f, _ in plain)
    for timed in (True, False):
        for a, b in zip(_run(_case(S, 0.01), kind, budget, timed), plain):
            assert a[:2] == b[:2]
            for n in b[2]:
                assert np.array_equal(a[2][n], b[2][n], equal_nan=True), (n, timed)
            assert np.array_equal(a[3], b[3], equal_nan=True)


def test_a_pool_in_recession_equals_each_alone():
    """Both kinds of pool kernels (common and own constants), through the event."""
    from swehr_b200.lib import Pool, Simulation
    cases = [_case(S, 0.01) for S in (1, 7, 5)]
    for c in cases:
        c.params["tend"] = 12.0
    other = _case(3, 0.01)
    other.params.update(tend=12.0, cohesion=5.0)
    for group in (cases, cases + [other]):
        with Pool(max_classes=8) as pool:
            scs = [pool.submit(c) for c in group]
            rng = np.random.default_rng(3)
            us = [_settled(c.sclass, "decaying", rng, (c.nx, c.ny)) for c in group]
            hs = [rng.uniform(2e-3, 6e-3, (c.nx, c.ny)) for c in group]
            for sc, u, h in zip(scs, us, hs):
                _write(sc, "h", h)
                for k, a in enumerate(u):
                    _write(sc, "U", a, k + 1)
            pool.run(-1)
            got = [sc.fields() for sc in scs]
        for c, u, h, g in zip(group, us, hs, got):
            with Simulation(c) as s:
                s.write_field("h", h)
                for k, a in enumerate(u):
                    s.write_field("U", a, k + 1)
                s.advance()
                want = s.fields()
            for n in want:
                assert np.array_equal(g[n], want[n], equal_nan=True), n


def _write(sc, name, arr, k=0):
    from swehr_b200.lib import FIELD_NAMES
    a = np.ascontiguousarray(arr)
    assert sc.L.swehr_write_field(sc.ctx, FIELD_NAMES[name], k, a.ctypes.data) == 0


@pytest.mark.parametrize("budget", [False, True], ids=["", "budget"])
def test_a_step_of_the_recession_takes_no_longer_than_one_of_the_rain(budget):
    """The 200 x 50 hillslope, whose coarse classes settle from step 2,900 on
    (two thirds of the warps at 3,800 hold a U_k below 2^-300) while it still
    flows.  Measured 1.07 (with budgets 1.05) times the time of a step in the
    rain; 2.4 (2.0) with every such cell computed twice."""
    from swehr_b200.lib import Simulation
    with Simulation(W.hillslope200x50(), budget=budget) as s:
        s.advance(max_steps=1500)
        rain = s.advance(max_steps=900)
        s.advance(max_steps=1030)
        after = s.advance(max_steps=700)
    ratio = (after.device_ms / after.steps_this_call) / (rain.device_ms / rain.steps_this_call)
    assert ratio < 1.35, ratio


@pytest.mark.parametrize("timed", [False, True], ids=["", "timed"])
@pytest.mark.parametrize("kind", ["storm", "film"])
def test_exponents_below_minus_700_equal_the_oracle(kind, timed):
    """Cells up to 75 radii from a storm's centre, and classes that settle out of a
    film of 1e-8 m within a step: exp through the subnormals to zero."""
    from harness import CLASS_FIELDS, STATE_FIELDS, OracleRun, compare
    from swehr_b200.lib import Simulation
    over = dict(hfilm=1e-8) if kind == "film" else dict(storm_peak=2e-4, storm_radius=0.2, storm_x0=5.0, storm_y0=6.0,
                                                         storm_vx=0.05, storm_vy=0.02)
    case = W.tiny_case(nx=20, ny=40, S=4, seed=12, rain_mmh=200.0, tend=1e3, **over)
    o = OracleRun(case, "shim")
    with Simulation(case) as s:
        s.set_timing(timed)
        for _ in range(4):
            o.advance(max_steps=60)
            pr = s.advance(max_steps=60)
            assert pr.t == o.t
            res = compare(s.fields(), o.fields(), STATE_FIELDS + CLASS_FIELDS)
            assert all(v[2] for v in res.values()), {k: v for k, v in res.items() if not v[2]}
