"""The count of launches when several threads step and run engines at once: what one thread
captures does not take in what the others launch meanwhile.  Each thread's work alone, times
the threads.  Tolerance zero."""
import threading

import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu

THREADS = 6


def work():
    for seed in range(12):
        p = make_params(max_days=9, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                        people_scaling=0.01, location_scaling=0.01)
        sim = pt.PandemicSim(p, seed)
        sim.setupSim()
        for _ in range(3):
            while sim.step_day()[0] != pt.PT_FINISHED:
                pass
            sim.reset_epidemic()
            sim.runToCompletion()
            sim.reset_epidemic()
        sim.close()


def test_count_is_the_sum_of_the_threads(native_lib):
    work()
    before = pt.launch_count()
    work()
    alone = pt.launch_count() - before
    threads = [threading.Thread(target=work) for _ in range(THREADS)]
    before = pt.launch_count()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert pt.launch_count() - before == THREADS * alone
