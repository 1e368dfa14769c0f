"""The fused hidden layers (k_umma_hidden) and the mean layer's direct output, at the edges
of their tiles: one to nine tiles of 128 rows, chunks that end inside a tile, each hidden width the kernel takes, input widths in both operand layouts
and over one K slice, one to four layers, one to eight networks.

Against the layer-by-layer kernels: a network whose hidden layers run fused gives bit for bit
what the same network gives when its batch goes through another number of rows, and the
FP64 network of test_gpu_tcgen05 within its tolerance (2e-2 of the largest output, 2e-3 on
average: BF16 activations)."""
import numpy as np
import pytest

from pandemicthrust_gb300 import surrogate as sg
from test_gpu_tcgen05 import reference_forward  # noqa: E402

pytestmark = pytest.mark.gpu


def network(widths, seed, max_batch):
    net = sg.MLP(widths, max_batch=max_batch, seed=seed)
    p = net.get_params()
    p = (p + np.random.default_rng(seed).standard_normal(p.shape) * 0.05).astype(np.float32)
    net.set_params(p)
    return net, p


@pytest.mark.parametrize("widths", [[11, 256, 222], [11, 256, 256, 256, 256, 222], [16, 64, 64, 7], [40, 128, 128, 96],
                                    [64, 192, 192, 192, 33], [200, 256, 256, 256], [1, 64, 1]])
def test_fused_layers_match_fp64_at_every_row_count(native_lib, widths):
    net, p = network(widths, 9, 1024)
    X = np.random.default_rng(3).uniform(-1, 1, (1100, widths[0])).astype(np.float32)
    whole = net.predict(X)   # a chunk of 1024 rows and one of 76
    ref = reference_forward(p, widths, X)
    scale = np.abs(ref).max()
    assert np.isfinite(whole).all()
    assert np.abs(whole - ref).max() <= 2e-2 * scale and np.abs(whole - ref).mean() <= 2e-3 * scale
    for rows in (1, 31, 127, 128, 129, 255, 256, 257, 384, 513):
        assert np.array_equal(net.predict(X[:rows]), whole[:rows]), rows
    net.close()


@pytest.mark.parametrize("members", [1, 2, 3, 5, 8])
def test_members_share_a_launch(native_lib, members):
    s = sg.Surrogate(1_000_000, hidden=128, depth=3, seed=5, members=members, max_batch=600)
    rng = np.random.default_rng(members)
    for net in s.nets:
        p = net.get_params()
        net.set_params((p + rng.standard_normal(p.shape) * 0.05).astype(np.float32))
    X = sg.features(sg.sample_scenarios(901, rng))
    y = s.raw_features(X)
    each = np.mean([net.predict(X).astype(np.float64) for net in s.nets], axis=0)
    # the same activations; FP32 sums of 128 x members terms in another order
    assert np.abs(y - each).max() <= 1e-5 * np.abs(each).max()
    # a changed member is packed again
    p = s.nets[-1].get_params()
    s.nets[-1].set_params((p * np.float32(0.5)).astype(np.float32))
    z = s.raw_features(X)
    each = np.mean([net.predict(X).astype(np.float64) for net in s.nets], axis=0)
    assert np.abs(z - each).max() <= 1e-5 * np.abs(each).max() and not np.array_equal(y, z)
    s.close()


def test_a_captured_call_has_the_weights_of_its_replay(native_lib):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    rng = np.random.default_rng(4)
    net = sg.MLP([11, 128, 128, 222], max_batch=512, seed=3, stream=stream.cuda_stream)
    s = sg.Surrogate.__new__(sg.Surrogate)
    s.nets = [net]
    x = torch.from_numpy(rng.uniform(-1, 1, (300, 11)).astype(np.float32)).cuda()
    y = torch.zeros(300, 222, device="cuda")
    torch.cuda.synchronize()
    s.raw_device(x.data_ptr(), 300, y.data_ptr())
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        s.raw_device(x.data_ptr(), 300, y.data_ptr())
    p = net.get_params()
    for seed in (1, 2):
        net.set_params((p + np.random.default_rng(seed).standard_normal(p.shape) * 0.05).astype(np.float32))
        y.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), net.predict(x.cpu().numpy())), seed
    net.close()
