"""Operands that the FP64 form's branch-free sequences do not take -- below
2^-300, subnormal, above 2^300, infinite, NaN, negative depths -- give the plain
operators' results: the face, cell or wave vector that meets one is computed
again.

The plain operators are reached without the sequences by a constant outside
their range that enters no result: the stream-power fraction F = 2^101 with
critical powers that no flow exceeds."""
import numpy as np
import pytest

from harness import OracleRun
from swehr_b200 import workloads as W

pytestmark = pytest.mark.gpu

TINY, HUGE = 2.0 ** -301, 2.0 ** 302
ODD = {
    "tiny": [TINY, 1e-200, 1e-300],
    "subnormal": [5e-324, 1e-310, -1e-315],
    "huge": [HUGE, 1e120, 1e160],
    "infinite": [np.inf, 1e308],
    "nan": [np.nan],
    "negative": [-1e-3, -0.0, -1e-12],
}
FIELDS = ("h", "hu", "hv", "U", "M", "totm", "totsed", "dep", "vinf")


def _fields(case, F, name, values, timed):
    from swehr_b200.lib import Simulation
    c = W.Case(case.name, dict(case.params, F=F, uc=1e300, uc2=1e300), case.topo, case.rain, case.ds, case.pfrac, case.ks)
    rng = np.random.default_rng(1)
    out = []
    with Simulation(c) as s:
        s.set_timing(timed)
        s.advance(max_steps=40)
        for n in ("h", "hu", "hv"):                   # moving water everywhere
            s.write_field(n, {"h": 2e-3, "hu": 1e-4, "hv": -5e-5}[n] * rng.uniform(0.5, 1.5, (c.nx, c.ny)))
        k = 2 if name in ("U", "M") else 0
        a = s.field(name, k)
        a[rng.random(a.shape) < 0.05] = rng.choice(values)
        s.write_field(name, a, k)
        for _ in range(3):
            pr = s.advance(max_steps=1)
            out.append((pr.t, pr.dt, pr.status, s.fields()))
    return out


@pytest.mark.parametrize("odd", list(ODD))
@pytest.mark.parametrize("name", FIELDS)
def test_odd_states_equal_the_plain_operators(name, odd):
    case = W.tiny_case(nx=21, ny=43, S=3, seed=8, rain_mmh=300.0, tend=1e4)
    plain = _fields(case, 2.0 ** 101, name, ODD[odd], True)
    for timed in (True, False):
        fast = _fields(case, 0.01, name, ODD[odd], timed)
        for a, b in zip(fast, plain):
            assert np.array_equal(np.array(a[:3], float), np.array(b[:3], float), equal_nan=True)
            for n in b[3]:
                assert np.array_equal(a[3][n], b[3][n], equal_nan=True), (n, timed)


def test_suspended_mass_decaying_to_zero_equals_the_oracle():
    """After the rain the coarse classes settle by many powers of ten a step,
    through the range the sequences refuse and the subnormals to zero."""
    from swehr_b200.lib import Simulation
    case = W.tiny_case(nx=16, ny=40, S=6, seed=9, rain_mmh=400.0, tend=90.0, uc=1e9, uc2=1e9)
    o = OracleRun(case, "shim")
    o.advance(t_stop=60.0)
    seen = 0
    with Simulation(case) as s:
        s.advance(t_stop=60.0)
        for _ in range(260):
            s.advance(max_steps=1)
            o.advance(max_steps=1)
            U, V = s.fields(("U",))["U"], o.fields()["U"]
            assert np.array_equal(U, V)
            seen += int(((U > 0) & (U < TINY)).sum())
    assert seen > 0
