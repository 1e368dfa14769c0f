"""The radix sort behind every bucket table, through pt_bucket_table_static: entry counts
at the edges of its 4096-entry tiles, bucket counts at the edges of its digits (one to
three passes of 1 to 8 bits), keys that are spread, equal, few, or sorted backwards.
The table is NumPy's stable argsort: whole numbers, tolerance zero."""
import ctypes

import numpy as np
import pytest

import pandemicthrust_gb300 as pt

pytestmark = pytest.mark.gpu


def keys_of(kind, n, buckets, rng):
    if kind == "spread":
        k = rng.integers(0, buckets, n)
    elif kind == "one":
        k = np.full(n, buckets - 1)
    elif kind == "few":
        k = rng.choice(rng.integers(0, buckets, 3), n)
    else:
        k = np.sort(rng.integers(0, buckets, n))[::-1]
    return np.ascontiguousarray(k, np.int32)


@pytest.mark.parametrize("buckets", [1, 2, 17, 256, 257, 5434, 65_536, 65_537, 1 << 20])
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 12_293, 300_001, 1 << 20])
def test_table_equals_stable_argsort(native_lib, n, buckets):
    torch = pytest.importorskip("torch")
    lib = pt.load_library()
    rng = np.random.default_rng(n * 31 + buckets)
    for kind in ("spread", "one", "few", "backwards"):
        k = keys_of(kind, n, buckets, rng)
        dk = torch.from_numpy(k).cuda()
        off = torch.full((buckets + 1,), -1, dtype=torch.int32, device="cuda")
        tab = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = lib.pt_bucket_table_static(ctypes.c_void_p(dk.data_ptr()), n, buckets, ctypes.c_void_p(off.data_ptr()),
                                        ctypes.c_void_p(tab.data_ptr()), None)
        assert rc == pt.PT_OK
        assert np.array_equal(tab.cpu().numpy(), np.argsort(k, kind="stable")), kind
        want = np.concatenate([[0], np.cumsum(np.bincount(k, minlength=buckets))])
        assert np.array_equal(off.cpu().numpy(), want), kind
