"""The per-person state asked for where the call may not wait (inside a capture of the
engine's stream, beside one of another stream): refused, with the caller's arrays as they
were.  Afterwards the state is that of an undisturbed engine.  Tolerance zero."""
import ctypes

import numpy as np
import pytest

import pandemicthrust_gb300 as pt
from oracle.oracle import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [True, False])
def test_refused_state_leaves_the_arrays_alone(native_lib, own):
    torch = pytest.importorskip("torch")
    p = make_params(max_days=4, r_pandemic=1.8, r_seasonal=1.5, initial_pandemic=20, initial_seasonal=20,
                    people_scaling=0.01, location_scaling=0.01)
    stream = torch.cuda.Stream()
    sim = pt.PandemicSim(p, 5, stream=stream.cuda_stream)
    sim.setupSim()
    sim.runToCompletion()
    want = sim.person_state()
    n = sim.info()["number_people"]
    arrays = [np.full(n, 77, np.uint8) for _ in range(7)]
    u8 = ctypes.POINTER(ctypes.c_uint8)
    rc, x = 0, torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    try:
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream if own else torch.cuda.Stream()):
            x += 1
            rc = sim.lib.pt_get_person_state(sim.h, *[a.ctypes.data_as(u8) for a in arrays])
    except RuntimeError:
        pass   # (a refusal may end the capture)
    torch.cuda.synchronize()
    assert rc < 0 and all((a == 77).all() for a in arrays)
    got = sim.person_state()
    assert all(np.array_equal(got[k], want[k]) for k in want)
    sim.close()
