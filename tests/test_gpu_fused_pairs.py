"""The fused hidden layers with several pairs of items a CTA: three pairs and more, an odd last
item and a last tile that is not full, at every hidden width and depth where a slot is used
again.  Bit for bit against the same rows in chunks of one item a CTA, and, where a network can
be written with an uneven hidden width (zero weights in the columns added, which the fused
layers do not take), against the layer-by-layer kernels: added zeros change no sum.  And
against the mma.sync path, whose sums run in another order: twice the 2e-2 / 2e-3 of the
largest output that test_gpu_tcgen05 allows either from the FP64 network (BF16 activations)."""
import numpy as np
import pytest

from pandemicthrust_gb300 import surrogate as sg

pytestmark = pytest.mark.gpu


def sms():
    return pytest.importorskip("torch").cuda.get_device_properties(0).multi_processor_count


def parameters(widths, seed):
    rng = np.random.default_rng(seed)
    return [(rng.uniform(-1, 1, (b, a)).astype(np.float32) * np.float32((6.0 / a) ** 0.5),
             rng.normal(0, 0.05, b).astype(np.float32)) for a, b in zip(widths[:-1], widths[1:])]


def network(layers, max_batch):
    net = sg.MLP([layers[0][0].shape[1]] + [w.shape[0] for w, _ in layers], max_batch=max_batch)
    net.set_params(np.concatenate([np.concatenate([w.ravel(), b]) for w, b in layers]))
    return net


def padded(layers, extra):
    """The same network with `extra` more columns in its last hidden layer, all weights to and from them zero."""
    (w, b), (v, c) = layers[-2:]
    return layers[:-2] + [(np.concatenate([w, np.zeros((extra, w.shape[1]), np.float32)]),
                           np.concatenate([b, np.zeros(extra, np.float32)])),
                          (np.concatenate([v, np.zeros((v.shape[0], extra), np.float32)], axis=1), c)]


@pytest.mark.parametrize("widths", [[16, 64, 64, 7], [11, 64, 64, 9], [11, 64, 64, 64, 9], [64, 64, 64, 5], [11, 64, 222],
                                    [3, 64, 64, 64, 64, 8], [11, 128, 128, 24], [40, 192, 192, 192, 17],
                                    [11, 256, 256, 222], [200, 256, 256, 256, 256, 33]])
def test_many_pairs_equal_one_item_a_cta(native_lib, widths):
    n = sms()
    rows = 128 * (6 * n + 3) - 51    # three pairs for every CTA, and a fourth with one item
    X = np.random.default_rng(rows).uniform(-1, 1, (rows, widths[0])).astype(np.float32)
    layers = parameters(widths, 5)
    fused, small = network(layers, rows), network(layers, 128 * n)
    y = fused.predict(X)
    assert np.array_equal(y, small.predict(X))
    small.close()
    if widths[-2] < 256 and len(widths) > 3:
        apart = network(padded(layers, 32), rows)
        assert np.array_equal(y, apart.predict(X))
        apart.close()
    fused.set_tcgen05(False)
    z = fused.predict(X)
    scale = np.abs(z).max()
    assert np.abs(y - z).max() <= 4e-2 * scale and np.abs(y - z).mean() <= 4e-3 * scale
    fused.close()


@pytest.mark.parametrize("members,hidden,depth", [(3, 64, 2), (8, 64, 2), (8, 128, 3), (4, 256, 4)])
def test_many_pairs_of_several_networks(native_lib, members, hidden, depth):
    n = sms()
    tiles = (6 * n) // members + 2
    rows = 128 * tiles - 77
    X = np.random.default_rng(members).uniform(-1, 1, (rows, 11)).astype(np.float32)
    got = []
    for chunk in (rows, 128 * (n // members)):
        s = sg.Surrogate(1_000_000, hidden=hidden, depth=depth, members=members, max_batch=chunk)
        for k, net in enumerate(s.nets):
            net.set_params(np.concatenate([np.concatenate([w.ravel(), b]) for w, b in parameters(net.widths, k)]))
        got.append(s.raw_features(X))
        s.close()
    assert np.array_equal(*got)
