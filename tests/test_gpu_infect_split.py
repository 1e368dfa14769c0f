"""Days on both sides of the line between eight lanes an infector and one thread an
infector (128 infectors an SM): the infected list grows past it during the run.  Against
the oracle, and against the run that has eight lanes on every day.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seeds,blocks", [(9_000, 8), (9_700, 1)])
def test_the_list_grows_past_the_line(native_lib, oracle_built, seeds, blocks):
    p = make_params(max_days=9, r_pandemic=2.0, r_seasonal=1.7, initial_pandemic=seeds, initial_seasonal=seeds,
                    people_scaling=0.1, location_scaling=0.1)
    o = Oracle(p, 31)
    o.setup()
    rows = []
    for coop in (0, 1):
        sim = pt.PandemicSim(p, 31)
        sim.set_tuning(dict(sim.tuning(), infect_coop=coop, infect_blocks_per_sm=blocks))
        sim.setupSim()
        limit = 128 * sim.info()["sm_count"]
        counts, infected = sim.runToCompletion()
        rows.append((counts, infected, sim.person_state()))
        sim.close()
    assert infected.min() <= limit < infected.max()
    for c, i in zip(*rows[0][:2]):
        _, oc, oi = o.step_day()
        assert list(c) == list(oc) and i == oi
    v = o.view()
    for k in ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s"):
        assert np.array_equal(rows[0][2][k], v[k]) and np.array_equal(rows[1][2][k], v[k]), k
    assert np.array_equal(rows[0][0], rows[1][0]) and np.array_equal(rows[0][1], rows[1][1])
    o.close()
