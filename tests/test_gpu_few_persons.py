"""The per-person state on both sides of the line (49,152 persons) between the host and the device
taking its words apart, all arrays and one at a time, alone and out of a batch.  The
oracle's state.  Tolerance zero."""
import ctypes

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu

FIELDS = ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s", "age")


@pytest.mark.parametrize("scale", [0.00002, 0.0207, 0.0211])
def test_state_on_both_sides(native_lib, oracle_built, scale):
    p = make_params(max_days=3, r_pandemic=2.0, r_seasonal=1.7, initial_pandemic=5, initial_seasonal=6,
                    people_scaling=scale, location_scaling=scale)
    o = Oracle(p, 3)
    o.setup()
    for _ in range(3):
        o.step_day()
    v = o.view()
    n = v["N"]
    assert scale < 0.02 or (n <= 49152) == (scale < 0.021)
    batch = pt.PandemicBatch([p, p], [8, 3])
    batch.setup()
    batch.run()
    sim = pt.PandemicSim(p, 3)
    sim.setupSim()
    sim.runToCompletion()
    for state in (sim.person_state(), batch.person_state(1)):
        for k in FIELDS:
            assert np.array_equal(state[k], v[k]), k
    u8 = ctypes.POINTER(ctypes.c_uint8)
    for j, k in enumerate(FIELDS):
        one = np.full(n + 8, 77, np.uint8)
        args = [None] * 7
        args[j] = one.ctypes.data_as(u8)
        assert sim.lib.pt_get_person_state(sim.h, *args) == 0
        assert np.array_equal(one[:n], v[k]) and (one[n:] == 77).all()
    sim.close()
    batch.close()
    o.close()
