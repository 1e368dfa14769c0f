"""What follows days that were queued by a call that was not allowed to wait (beside another
stream's capture): steps after a refused run, a run after a refused step, either after
some days, on epidemics that last and that end.  Row by row those of an undisturbed
engine, with its return codes.  Tolerance zero."""
import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu


def params(r):
    return make_params(max_days=14, r_pandemic=r, r_seasonal=r, initial_pandemic=20, initial_seasonal=20,
                       people_scaling=0.01, location_scaling=0.01)


def steps(sim):
    out = []
    while True:
        rc, c, i = sim.step_day()
        if rc == pt.PT_FINISHED:
            return out
        out.append((rc, list(c), i))
        if rc == pt.PT_DONE:
            return out


def refused(call):
    torch = pytest.importorskip("torch")
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            x += 1
            with pytest.raises(pt.PtError):
                call()
    except RuntimeError:
        pass   # (a refusal ends the capture too)
    torch.cuda.synchronize()


@pytest.mark.parametrize("r", [1.8, 0.0])
@pytest.mark.parametrize("before", [0, 2])
@pytest.mark.parametrize("first,then", [("run", "steps"), ("step", "run"), ("step", "steps"), ("run", "run")])
def test_days_after_a_refusal(native_lib, r, before, first, then):
    sim = pt.PandemicSim(params(r), 5)
    sim.setupSim()
    want = steps(sim)
    assert (want[-1][0] == pt.PT_DONE) == (r == 0.0)
    for _ in range(2):   # (the second time with the graphs made)
        sim.reset_epidemic()
        got = [sim.step_day() for _ in range(before)]
        got = [(rc, list(c), i) for rc, c, i in got]
        refused(sim.runToCompletion if first == "run" else sim.step_day)
        if then == "steps":
            assert got + steps(sim) == want
        else:
            c, i = sim.runToCompletion()
            assert c.tolist() == [w[1] for w in want] and i.tolist() == [w[2] for w in want]
        assert sim.step_day()[0] == (pt.PT_DONE if r == 0.0 else pt.PT_FINISHED)
    sim.close()
