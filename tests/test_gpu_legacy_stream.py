"""Runs and steps on the legacy default stream, which cannot be captured: queued day by day,
call after call, with the rows of an engine on its own stream.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu

LEGACY = 1   # cudaStreamLegacy


def rows_of(sim, runs_from):
    """The rows of `runs_from` stepped days, then a run."""
    for _ in range(runs_from):
        sim.step_day()
    c, i = sim.runToCompletion()
    return np.concatenate([c, i[:, None]], axis=1)


@pytest.mark.parametrize("order", [(0, 0, 3), (3, 0), (2, 9, 0)])
def test_rows_are_those_of_an_own_stream(native_lib, order):
    p = make_params(max_days=9, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                    people_scaling=0.01, location_scaling=0.01)
    own = pt.PandemicSim(p, 5)
    own.setupSim()
    want = rows_of(own, 0)
    sim = pt.PandemicSim(p, 5, stream=LEGACY)
    sim.setupSim()
    for steps in order:
        assert np.array_equal(rows_of(sim, steps), want)
        a, b = sim.person_state(), own.person_state()
        assert all(np.array_equal(a[k], b[k]) for k in b)
        sim.reset_epidemic()
    sim.close()
    own.close()
