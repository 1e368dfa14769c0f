"""Engines made, stepped and run in two threads while a third waits for the whole device over and
over, which is forbidden while any stream is being captured: nobody is refused, and the
rows are an undisturbed engine's.  Tolerance zero."""
import threading

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu

PARAMS = make_params(max_days=9, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                     people_scaling=0.01, location_scaling=0.01)


def rows(core):
    """Stepped rows and a run's, the second time from the graphs, and again with complete tables."""
    sim = pt.PandemicSim(PARAMS, core)
    sim.setupSim()
    out = []
    for _ in range(2):
        for full in (False, True):
            sim.set_full_tables(full)
            while True:
                rc, c, i = sim.step_day()
                if rc == pt.PT_FINISHED:
                    break
                out.append(list(c) + [i])
            sim.reset_epidemic()
            for _ in range(2):
                c, i = sim.runToCompletion()
                out += np.concatenate([c, i[:, None]], axis=1).tolist()
                sim.reset_epidemic()
    sim.close()
    return out


def test_waits_for_the_device_do_not_matter(native_lib):
    torch = pytest.importorskip("torch")
    torch.zeros(1, device="cuda")
    want = [rows(core) for core in range(3)]
    assert all(w[:9] == w[9:18] for w in want)
    bad, done = [], threading.Event()

    def work(first):
        try:
            for j in range(12):
                assert rows((first + j) % 3) == want[(first + j) % 3]
        except BaseException as e:   # reported by the test's thread
            bad.append(e)

    def wait():
        try:
            while not done.is_set():
                torch.cuda.synchronize()
        except BaseException as e:
            bad.append(e)

    workers = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    waiter = threading.Thread(target=wait)
    for t in workers + [waiter]:
        t.start()
    for t in workers:
        t.join()
    done.set()
    waiter.join()
    assert not bad, bad
