"""The one-launch infected list and marks of small runs (up to 1024 person tiles) on both
sides of their limits, against the oracle, weekdays and a weekend: populations just below
and just above the limit, one tile, and a weekend bitmap just below and above the words
that are marked in shared memory.  Then a batch whose instances end on different days,
each against its own single run.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu

FIELDS = ("status_p", "status_s", "day_p", "day_s", "gen_p", "gen_s")


@pytest.mark.parametrize("scale,loc,seeds,days", [(1.775, 1.775, 300, 7), (1.79, 1.79, 300, 7), (0.0015, 0.0015, 40, 9),
                                                  (0.05, 1.0, 900, 8), (0.05, 4.0, 900, 8)])
def test_small_runs_equal_the_oracle(native_lib, oracle_built, scale, loc, seeds, days):
    p = make_params(max_days=days, r_pandemic=2.0, r_seasonal=1.7, initial_pandemic=seeds, initial_seasonal=seeds,
                    people_scaling=scale, location_scaling=loc)
    sim = pt.PandemicSim(p, 12)
    sim.setupSim()
    o = Oracle(p, 12)
    o.setup()
    counts, infected = sim.runToCompletion()
    for c, i in zip(counts, infected):
        _, oc, oi = o.step_day()
        assert list(c) == list(oc) and i == oi
    st, v = sim.person_state(), o.view()
    for k in FIELDS:
        assert np.array_equal(st[k], v[k]), k
    o.close()
    sim.close()


def test_instances_that_end_on_different_days(native_lib):
    params = [make_params(max_days=days, r_pandemic=r, r_seasonal=r, initial_pandemic=s, initial_seasonal=s,
                          people_scaling=scale, location_scaling=scale)
              for days, r, s, scale in ((20, 1.9, 30, 0.01), (6, 1.5, 5, 0.002), (40, 0.05, 3, 0.004), (33, 1.2, 1, 0.006))]
    batch = pt.PandemicBatch(params, [7, 8, 9, 10])
    batch.setup()
    batch.run()
    for k, p in enumerate(params):
        sim = pt.PandemicSim(p, 7 + k)
        sim.setupSim()
        counts, infected = sim.runToCompletion()
        bc, bi = batch.counts(k)
        assert np.array_equal(counts, bc) and np.array_equal(infected, bi)
        sim.close()
    batch.close()


def test_a_run_inside_a_capture_is_refused(native_lib):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    p = make_params(max_days=4, r_pandemic=1.5, r_seasonal=1.5, initial_pandemic=5, initial_seasonal=5,
                    people_scaling=0.002, location_scaling=0.002)
    sim = pt.PandemicSim(p, 3, stream=stream.cuda_stream)
    sim.setupSim()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        with pytest.raises(pt.PtError):
            sim.runToCompletion()
        with pytest.raises(pt.PtError):
            sim.step_day()
    counts, infected = sim.runToCompletion()
    other = pt.PandemicSim(p, 3)
    other.setupSim()
    c, i = other.runToCompletion()
    assert np.array_equal(counts, c) and np.array_equal(infected, i)
    sim.close()
    other.close()
