"""A call that a capture in another thread refuses, and the same thread's next calls when the
capture is over: they work (the refused call's error is not reported again by the next
launch) and give what an undisturbed engine and network give.  Tolerance zero."""
import threading

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params
from pandemicthrust_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu


def run(sim):
    sim.reset_epidemic()
    c, i = sim.runToCompletion()
    return c.tolist(), i.tolist()


@pytest.mark.parametrize("kind", ["engine", "network"])
def test_the_next_call_works(native_lib, kind):
    torch = pytest.importorskip("torch")
    p = make_params(max_days=6, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                    people_scaling=0.01, location_scaling=0.01)
    X = np.random.default_rng(0).uniform(-1, 1, (200, 11)).astype(np.float32)
    sim = pt.PandemicSim(p, 5)
    sim.setupSim()
    stream = torch.cuda.Stream()
    net = sg.MLP([11, 64, 64, 5], max_batch=256, stream=stream.cuda_stream)
    want = (run(sim), net.predict(X).tolist())
    sim.reset_epidemic()
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    begun, over, got, refusals = threading.Event(), threading.Event(), [], []

    def work():
        begun.wait(20)
        try:
            sim.step_day() if kind == "engine" else net.predict(X)
        except pt.PtError as e:
            refusals.append(e)
        over.set_me.set()
        over.wait(20)
        try:
            got.append((run(sim), net.predict(X).tolist()))
        except pt.PtError as e:
            got.append(e)

    over.set_me = threading.Event()   # the refused call has returned
    t = threading.Thread(target=work)
    t.start()
    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode="global"):
            x += 1
            begun.set()
            over.set_me.wait(20)
    except RuntimeError:
        pass   # (a refusal ends the capture too)
    torch.cuda.synchronize()
    over.set()
    t.join()
    assert refusals and got == [want]
    sim.close()
    net.close()
