"""Marking into a bitmap that no block's shared memory holds (above 8192 words) while the
infected are at least 32 to a word: the run equals one that materialises every bucket.
Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loc", [22.0, 24.0])
def test_marks_looked_at_before_they_are_set(native_lib, loc):
    p = make_params(max_days=7, r_pandemic=200.0, r_seasonal=100.0, initial_pandemic=9000, initial_seasonal=9000,
                    people_scaling=1.8, location_scaling=loc)
    runs = []
    for full in (False, True):
        sim = pt.PandemicSim(p, 21)
        sim.setupSim()
        sim.set_full_tables(full)
        counts, infected = sim.runToCompletion()
        info = sim.info()
        runs.append((counts, infected, sim.person_state()))
        sim.close()
    places = sum(info["type_count"][9:])   # weekend errands: ten hours of them
    words = 10 * places // 32 + 1
    assert words > 8192 and infected[5:].min() >= 32 * words
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    for k in ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s"):
        assert np.array_equal(runs[0][2][k], runs[1][2][k]), k
