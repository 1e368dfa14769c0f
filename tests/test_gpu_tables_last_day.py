"""The day's tables after an epidemic has ended: the day that finds nobody infected builds none,
so keys, table and offsets stay those of the day before (of the same type).  Populations
with the one-launch infected list and with the three-launch form, stepped and run,
with complete tables and without.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,full", [(0.002, True), (0.05, False), (0.05, True), (1.82, False)])
def test_tables_stay(native_lib, scale, full):
    # nobody infects anybody: the seeds recover on day 10, a weekday like day 9
    p = make_params(max_days=14, r_pandemic=0.0, r_seasonal=0.0, initial_pandemic=40, initial_seasonal=40,
                    people_scaling=scale, location_scaling=scale)
    sim = pt.PandemicSim(p, 5)
    sim.setupSim()
    sim.set_full_tables(full)
    for day in range(10):
        rc, _, infected = sim.step_day()
        assert rc == pt.PT_OK and infected > 0
    before = sim.day_tables()
    rc, _, infected = sim.step_day()
    assert rc == pt.PT_DONE and infected == 0
    after = sim.day_tables()
    sim.reset_epidemic()
    sim.runToCompletion()
    run = sim.day_tables()
    sim.close()
    used = before["offsets"][-2] if full else before["offsets"][:-1].max()
    assert used > 0
    for t in (after, run):
        assert t["entries"] == before["entries"] and t["buckets"] == before["buckets"]
        assert np.array_equal(t["keys"], before["keys"]) and np.array_equal(t["offsets"], before["offsets"])
        assert np.array_equal(t["people"][:used], before["people"][:used])
