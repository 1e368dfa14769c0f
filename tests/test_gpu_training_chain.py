"""The chained training pass (k_chain) at its edges: batches around its 16 rows, widths
around a CTA's 64 columns and the 256 it takes, one to eight layers; and, with nine layers
or a width of 257, the layer-by-layer pass on the other side of the line.

Gradients against the FP64 network of test_gpu_surrogate: activations and dZ are rounded
to BF16 (2^-9 each) between layers, so a relative L2 error of 3e-2 as there, 6e-2 from
eight layers on (the roundings of twice as many layers)."""
import numpy as np
import pytest

from pandemicthrust_gb300 import surrogate as sg
from test_gpu_surrogate import reference_gradients  # noqa: E402

pytestmark = pytest.mark.gpu

SHAPES = [([256, 256], 1), ([17, 64, 65], 15), ([64, 16, 240, 16], 16), ([5, 63, 129, 2], 17), ([200, 72, 256, 250], 31),
          ([11, 40, 40, 40, 40, 40, 40, 40, 9], 50), ([11, 40, 40, 40, 40, 40, 40, 40, 40, 9], 50),
          ([11, 257, 20], 33), ([257, 20, 20], 33)]


@pytest.mark.parametrize("widths,batch", SHAPES)
def test_gradients(native_lib, widths, batch):
    rng = np.random.default_rng(sum(widths) + batch)
    net = sg.MLP(widths, max_batch=batch + 40, seed=3)
    p = net.get_params()
    p = (p + rng.normal(0, 0.05, p.size)).astype(np.float32)
    net.set_params(p)
    # a larger batch first: nothing of its rows may stay
    Xl = rng.uniform(-1, 1, (batch + 40, widths[0])).astype(np.float32)
    net.gradients(Xl, rng.normal(0, 1, (batch + 40, widths[-1])).astype(np.float32))
    X = rng.uniform(-1, 1, (batch, widths[0])).astype(np.float32)
    Y = rng.normal(0, 1, (batch, widths[-1])).astype(np.float32)
    g, loss = net.gradients(X, Y)
    ref, ref_loss = reference_gradients(p, widths, X, Y)
    assert abs(loss - ref_loss) <= 1e-2 * ref_loss
    tol = 3e-2 if len(widths) < 9 else 6e-2
    off = 0
    for l in range(len(widths) - 1):
        for n in (widths[l + 1] * widths[l], widths[l + 1]):
            a, b = g[off:off + n].astype(np.float64), ref[off:off + n]
            assert np.linalg.norm(a - b) <= tol * max(np.linalg.norm(b), 1e-30), (l, n)
            off += n
    net.close()
