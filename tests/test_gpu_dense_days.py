"""Days on which almost everyone infected infects: the claim queue of the infection
kernels (filled, overflowing, empty) and the marking of buckets through shared memory,
against the oracle.  A reproduction number of 400 makes nearly every contact a claim, so
a warp's round pushes several hundred; a large seed share makes the infected outnumber
the bitmap's words from the first day.  Tolerance zero: whole numbers."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu

FIELDS = ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s")
# (people_scaling, location_scaling, R, seeds a strain): overflowing queues; many
# infected on few buckets (shared marks); the same with a bitmap too large for them
CASES = [(0.004, 0.004, 400.0, 700), (0.1, 0.01, 1.6, 60_000), (0.1, 6.0, 1.6, 60_000)]


@pytest.mark.parametrize("scale,loc,r,seeds", CASES)
@pytest.mark.parametrize("coop", [0, 1])
def test_dense_days_equal_the_oracle(native_lib, oracle_built, scale, loc, r, seeds, coop):
    p = make_params(max_days=8, r_pandemic=r, r_seasonal=r / 2, initial_pandemic=seeds, initial_seasonal=seeds,
                    people_scaling=scale, location_scaling=loc)
    sim = pt.PandemicSim(p, 5)
    sim.setupSim()
    sim.set_tuning(dict(sim.tuning(), infect_coop=coop))
    o = Oracle(p, 5)
    o.setup()
    while True:
        rc, c, i = sim.step_day()
        orc, oc, oi = o.step_day()
        assert rc == orc
        if rc == 2:
            break
        assert c == oc and i == oi
        if rc == 1:
            break
    st, v = sim.person_state(), o.view()
    for k in FIELDS:
        assert np.array_equal(st[k], v[k]), k
    o.close()
    sim.close()
