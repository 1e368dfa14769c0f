"""The sweep's status counts where most persons are healthy, vaccinated or infected: every
person of a small population a seed, most of it vaccinated, populations that end inside a
thread's four persons, and a batch of many small instances whose blocks pass from one to
the next.  Against the oracle, and the batch against single runs.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import Oracle, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,seeds,core", [(0.002, 2000, 1), (0.002, 2000, 2), (0.003, 1, 3), (0.003, 1, 4), (0.05, 30_000, 5)])
def test_counts_equal_the_oracle(native_lib, oracle_built, scale, seeds, core):
    p = make_params(max_days=30, r_pandemic=1.9, r_seasonal=1.4, initial_pandemic=seeds, initial_seasonal=seeds // 2 + 1,
                    people_scaling=scale, location_scaling=scale)
    sim = pt.PandemicSim(p, core)
    sim.setupSim()
    o = Oracle(p, core)
    o.setup()
    counts, infected = sim.runToCompletion()
    n = sim.info()["number_people"]
    for c, i in zip(counts, infected):
        _, oc, oi = o.step_day()
        assert list(c) == list(oc) and i == oi
        assert sum(c[:8]) == n and sum(c[8:]) == n
    o.close()
    sim.close()


@pytest.mark.parametrize("instances,scale", [(6, 0.004), (3, 2.5)])
def test_instances_share_blocks(native_lib, instances, scale):
    params = [make_params(max_days=12, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=50, initial_seasonal=20,
                          people_scaling=scale * (1 + 0.1 * k), location_scaling=scale) for k in range(instances)]
    iv = dict(vaccination_coverage=0.6)
    batch = pt.PandemicBatch(params, list(range(40, 40 + instances)))
    batch.set_interventions([iv] * instances)
    batch.setup()
    batch.run()
    for k, p in enumerate(params):
        sim = pt.PandemicSim(p, 40 + k)
        sim.set_interventions(iv)
        sim.setupSim()
        counts, infected = sim.runToCompletion()
        bc, bi = batch.counts(k)
        assert np.array_equal(counts, bc) and np.array_equal(infected, bi)
        assert (counts.reshape(len(counts), 2, 8).sum(axis=2) == sim.info()["number_people"]).all()
        sim.close()
    batch.close()
