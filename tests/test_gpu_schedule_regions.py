"""The schedule kernel's regions against the oracle: populations below one region, odd
ones, ones that end inside a round, on and past person-tile boundaries, and one large
enough for wider regions; alone, with complete tables, and side by side in a batch.

Tolerance zero: the statistics rows and every person's state after nine days (both day
types) are whole numbers, and the schedule's keys and tables decide them."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu

FIELDS = ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s")
# people_scaling: about 30, 61, 130, 4,000, 8,300, 47,000 persons, and 4.2M
SCALES = [0.000013, 0.000026, 0.000055, 0.0017, 0.0035, 0.02, 1.8]
DAYS = 9


def params(scale):
    return make_params(max_days=DAYS, r_pandemic=2.1, r_seasonal=1.6, initial_pandemic=max(1, int(2000 * scale)),
                       initial_seasonal=max(1, int(1500 * scale)), people_scaling=scale, location_scaling=scale)


def oracle_run(p, seed):
    o = Oracle(p, seed)
    o.setup()
    rows = []
    for _ in range(DAYS):
        rc, c, i = o.step_day()
        if rc == 2:
            break
        rows.append((list(c), i))
        if rc == 1:
            break
    state = {k: np.array(v) for k, v in o.view().items() if k in FIELDS}
    o.close()
    return rows, state


def assert_rows(rows, counts, infected):
    assert len(rows) == len(infected)
    for d, (c, i) in enumerate(rows):
        assert counts[d].tolist() == c and infected[d] == i, d


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("full", [False, True])
def test_regions_equal_the_oracle(native_lib, oracle_built, scale, full):
    if full and scale > 1:
        pytest.skip("complete tables at one small size are enough")
    rows, state = oracle_run(params(scale), 41)
    sim = pt.PandemicSim(params(scale), 41)
    sim.setupSim()
    sim.set_full_tables(full)
    counts, infected = sim.runToCompletion()
    st = sim.person_state()
    sim.close()
    assert_rows(rows, counts, infected)
    for k in FIELDS:
        assert np.array_equal(st[k], state[k]), k


def test_uneven_instances_side_by_side_equal_the_oracle(native_lib, oracle_built):
    scales = SCALES[:6] * 2
    b = pt.PandemicBatch([params(s) for s in scales], [100 + k for k in range(len(scales))])
    b.setup()
    b.run()
    for k, s in enumerate(scales):
        rows, state = oracle_run(params(s), 100 + k)
        counts, infected = b.counts(k)
        assert_rows(rows, counts, infected)
        st = b.person_state(k)
        for f in FIELDS:
            assert np.array_equal(st[f], state[f]), (k, f)
    b.close()
