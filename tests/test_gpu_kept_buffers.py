"""The small host buffers that destroyed engines and networks leave for the next: engines of several
sizes stepped, networks trained and asked, made and closed by several threads at once, while
another thread hands the kept memory back.  Rows against an undisturbed run (tolerance zero),
predictions bit for bit."""
import threading

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params
from pandemicthrust_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu


def stepped(params):
    batch = pt.PandemicBatch(params, list(range(len(params))))
    batch.setup()
    for _ in range(6):
        batch.step_day()
    rows = [batch.counts(k) for k in range(len(params))]
    batch.close()
    return rows


def test_kept_buffers_between_threads(native_lib):
    p = [make_params(max_days=6, r_pandemic=1.5, r_seasonal=1.3, initial_pandemic=5, initial_seasonal=3,
                     people_scaling=0.0005 * (1 + k), location_scaling=0.001) for k in range(40)]
    sizes = (1, 7, 15, 40)
    X = np.random.default_rng(0).uniform(-1, 1, (200, 11)).astype(np.float32)

    def predicted(seed):
        net = sg.MLP([11, 64, 64, 5], max_batch=256, seed=seed)
        y = net.predict(X)
        net.gradients(X, y)
        net.close()
        return y

    want = {k: stepped(p[:k]) for k in sizes}
    ys = [predicted(s) for s in range(4)]
    bad, done = [], threading.Event()

    def work(seed):
        try:
            for j in range(8):
                k = sizes[(seed + j) % 4]
                for (c, i), (wc, wi) in zip(stepped(p[:k]), want[k]):
                    assert np.array_equal(c, wc) and np.array_equal(i, wi)
                assert np.array_equal(predicted((seed + j) % 4), ys[(seed + j) % 4])
        except BaseException as e:   # reported by the test's thread
            bad.append(e)

    def trim():
        while not done.wait(0.005):
            assert native_lib.pt_trim_device_memory() == 0

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    trimmer = threading.Thread(target=trim)
    for t in threads + [trimmer]:
        t.start()
    for t in threads:
        t.join()
    done.set()
    trimmer.join()
    assert not bad, bad
