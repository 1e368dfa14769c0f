"""A network is closed while another stream is being captured (a relaxed capture, which allows
waiting for a stream and freeing): the capture goes on and its graph does its work."""
import numpy as np
import pytest

from pandemicthrust_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own", [False, True])
def test_closing_does_not_end_the_capture(native_lib, own):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    net = sg.MLP([11, 64, 64, 5], max_batch=256, stream=stream.cuda_stream if own else None)
    net.predict(np.zeros((200, 11), np.float32))
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        x += 1
        net.close()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()
