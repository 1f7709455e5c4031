"""After a wait on the device gave up (its flag is set here from the host) no
further step is taken: swehr_advance returns SWEHR_TIMEOUT at once, on the many-
steps launches (small domains), on the two-kernel graph and on the timed path."""
import ctypes as C
import os

import numpy as np
import pytest

import swehr_b200
from swehr_b200 import workloads as W

pytestmark = pytest.mark.gpu

TIMEOUT = 3


@pytest.mark.parametrize("path", ["many_steps", "graph", "timed"])
def test_no_step_after_a_wait_gave_up(path):
    from swehr_b200.lib import Simulation, SwehrError
    probe = C.CDLL(os.path.join(os.path.dirname(swehr_b200.__file__), "libswehr_probe.so"))
    probe.swehr_probe_give_up.argtypes = [C.c_void_p]
    case = W.tiny_case(nx=20, ny=40, S=2, seed=4, rain_mmh=300.0, tend=1e4)
    with Simulation(case, budget=path == "graph") as s:       # budgets keep two kernels a step
        s.set_timing(path == "timed")
        assert s.advance(max_steps=5).steps == 5
        before = s.fields()
        assert probe.swehr_probe_give_up(s.ctx) == 0
        for steps in (-1, 300, -1):
            with pytest.raises(SwehrError) as err:
                s.advance(max_steps=steps)
            assert err.value.status == TIMEOUT
        after = s.fields()
        for n in before:
            assert np.array_equal(before[n], after[n], equal_nan=True), n
