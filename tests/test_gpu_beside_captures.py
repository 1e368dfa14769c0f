"""Days while another stream is being captured.  A capture that forbids its thread to wait
refuses them, before anything is queued: the run or the steps that follow give the rows of
an undisturbed run.  A relaxed capture does not forbid it, and the rows are right at once.
Against the same scenario's undisturbed run.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu

PARAMS = make_params(max_days=9, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                     people_scaling=0.01, location_scaling=0.01)


def rows_of_steps(sim):
    rows = []
    while True:
        rc, c, i = sim.step_day()
        if rc == pt.PT_FINISHED:
            return np.array(rows)
        rows.append(list(c) + [i])


def rows_of_run(sim):
    c, i = sim.runToCompletion()
    return np.concatenate([c, i[:, None]], axis=1)


@pytest.fixture(scope="module")
def want(native_lib):
    sim = pt.PandemicSim(PARAMS, 5)
    sim.setupSim()
    rows = rows_of_run(sim)
    sim.close()
    return rows


@pytest.mark.parametrize("days", [rows_of_run, rows_of_steps])
@pytest.mark.parametrize("mode", ["global", "thread_local"])
@pytest.mark.parametrize("before", [0, 3])
def test_refused_days_leave_nothing_behind(want, days, mode, before):
    torch = pytest.importorskip("torch")
    sim = pt.PandemicSim(PARAMS, 5)
    sim.setupSim()
    first = [sim.step_day() for _ in range(before)]
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    refused = False
    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode=mode):
            x += 1
            with pytest.raises(pt.PtError):
                days(sim)
            refused = True
    except RuntimeError:
        pass   # (a refusal ends the capture too)
    torch.cuda.synchronize()
    assert refused
    got = days(sim)
    if days is rows_of_steps and before:
        got = np.concatenate([[list(c) + [i] for _, c, i in first], got])
    assert np.array_equal(got, want)
    sim.close()


@pytest.mark.parametrize("days", [rows_of_run, rows_of_steps])
def test_a_relaxed_capture_does_not_matter(want, days):
    torch = pytest.importorskip("torch")
    sim = pt.PandemicSim(PARAMS, 5)
    sim.setupSim()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode="relaxed"):
        x += 1
        assert np.array_equal(days(sim), want)
    torch.cuda.synchronize()
    sim.reset_epidemic()
    assert np.array_equal(days(sim), want)
    sim.close()
