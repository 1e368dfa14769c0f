"""The training GEMMs at the edges of their 32 x 32 tiles, 16-term steps, 64-term stages and
512-row bias stages: widths of 1, odd, and past 256, one to four layers, batches of 1 and
not a multiple of anything.

Gradients against the FP64 network of test_gpu_surrogate (BF16 weights and inputs): the
kernels round activations and dZ to BF16 (2^-9 each) between layers, so a relative L2
error of 3e-2 as there.  One training step against Adam in FP64 on those gradients: FP32
arithmetic on values below 1, so 2e-6."""
import numpy as np
import pytest

from pandemicthrust_gb300 import surrogate as sg
from test_gpu_surrogate import reference_gradients  # noqa: E402

pytestmark = pytest.mark.gpu

SHAPES = [([1, 1], 1), ([3, 5], 33), ([11, 31, 7], 17), ([16, 33, 64, 100], 100), ([40, 300, 65, 24], 513),
          ([11, 256, 256, 256, 256, 222], 512), ([7, 48, 48, 48, 3], 1100)]


@pytest.mark.parametrize("widths,batch", SHAPES)
def test_gradients_and_one_step(native_lib, widths, batch):
    rng = np.random.default_rng(sum(widths) + batch)
    net = sg.MLP(widths, max_batch=batch + 3, seed=2)
    p = net.get_params()
    p = (p + rng.normal(0, 0.05, p.size)).astype(np.float32)
    net.set_params(p)
    # a larger batch first: its rows past `batch` must not leak into the next sums
    Xl = rng.uniform(-1, 1, (batch + 3, widths[0])).astype(np.float32)
    net.gradients(Xl, rng.normal(0, 1, (batch + 3, widths[-1])).astype(np.float32))
    X = rng.uniform(-1, 1, (batch, widths[0])).astype(np.float32)
    Y = rng.normal(0, 1, (batch, widths[-1])).astype(np.float32)
    g, loss = net.gradients(X, Y)
    ref, ref_loss = reference_gradients(p, widths, X, Y)
    assert abs(loss - ref_loss) <= 1e-2 * ref_loss
    off = 0
    for l in range(len(widths) - 1):
        for n in (widths[l + 1] * widths[l], widths[l + 1]):
            a, b = g[off:off + n].astype(np.float64), ref[off:off + n]
            assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-30), (l, n)
            off += n
    # one step over the whole data set: the rows' order only reorders the FP32 sums
    net.set_data(X, Y)
    net.train(1, batch=batch, lr=1e-3, seed=4)
    q = net.get_params().astype(np.float64)
    g64 = g.astype(np.float64)
    step = 1e-3 * g64 / (np.abs(g64) + 1e-8)    # Adam's first step: m / c1 = g, v / c2 = g^2
    big = np.abs(g64) > 1e-5                    # below, the sums' order decides the sign
    assert np.abs(q - (p - step))[big].max(initial=0) <= 2e-6
    assert np.abs(q - p).max() <= 1.001e-3 + 1e-6
    net.close()
