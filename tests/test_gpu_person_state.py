"""The per-person state as the device takes it apart: populations of every remainder of four,
one and several instances, and calls that ask for some of the arrays only.  Against the
oracle.  Tolerance zero."""
import ctypes

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu

FIELDS = ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s")


def params(scale):
    return make_params(max_days=3, r_pandemic=2.0, r_seasonal=1.7, initial_pandemic=20, initial_seasonal=30,
                       people_scaling=scale, location_scaling=scale)


@pytest.mark.parametrize("scale", [0.0006, 0.002, 0.05])
def test_state_equals_the_oracle_at_every_remainder(native_lib, oracle_built, scale):
    seen = set()
    cores = []
    for core in range(1, 60):
        sim = pt.PandemicSim(params(scale), core)
        sim.setupSim()
        n = sim.info()["number_people"]
        if n % 4 not in seen:
            seen.add(n % 4)
            cores.append(core)
            sim.runToCompletion()
            o = Oracle(params(scale), core)
            o.setup()
            for _ in range(3):
                o.step_day()
            st, v = sim.person_state(), o.view()
            for k in FIELDS:
                assert np.array_equal(st[k], v[k]), (core, k)
            u8 = ctypes.POINTER(ctypes.c_uint8)
            some = np.full(n + 8, 77, np.uint8)
            rc = sim.lib.pt_get_person_state(sim.h, None, None, some.ctypes.data_as(u8), None, None, None, None)
            assert rc == 0 and np.array_equal(some[:n], v["day_p"]) and (some[n:] == 77).all()
            o.close()
        sim.close()
        if len(seen) == 4:
            break
    assert len(seen) == 4
    batch = pt.PandemicBatch([params(scale)] * 4, cores)
    batch.setup()
    batch.run()
    for k, core in enumerate(cores):
        sim = pt.PandemicSim(params(scale), core)
        sim.setupSim()
        sim.runToCompletion()
        a, b = batch.person_state(k), sim.person_state()
        assert all(np.array_equal(a[f], b[f]) for f in FIELDS + ("age",))
        sim.close()
    batch.close()
