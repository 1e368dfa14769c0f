"""The rows of stepped days of batches whose rows fill one block, a block and a row more, and many
blocks (18 words an instance, 256 a block): each day's equal those of the same batch run
through.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instances", [14, 15, 57, 1001])
def test_rows_of_every_instance(native_lib, instances):
    params = [make_params(max_days=6 + k % 5, r_pandemic=1.2 + 0.1 * (k % 9), r_seasonal=1.3, initial_pandemic=1 + k % 7,
                          initial_seasonal=3, people_scaling=0.0002, location_scaling=0.001) for k in range(instances)]
    batch = pt.PandemicBatch(params, list(range(instances)))
    batch.setup()
    batch.run()
    want = [batch.counts(k) for k in range(instances)]
    for _ in range(2):   # (the second time from the captured days)
        batch.reset_epidemic()
        for _ in range(10):
            batch.step_day()
        for k in range(instances):
            c, i = batch.counts(k)
            assert np.array_equal(c, want[k][0]) and np.array_equal(i, want[k][1]), k
    batch.close()
