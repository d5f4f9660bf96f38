"""GPU: the bucketed sort where a record's word (low key bits, input index) is all
ones, as the padding of a bucket that is merge-sorted: 2^15 pairs of 53-bit
keys leave 49 key bits and 15 index bits, and the last pair has the largest
key.  60 equal keys crowd its bucket."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("crowd", [52, 55, 58, 60, 69])
def test_largest_word_is_not_taken_for_padding(cuda, torch, crowd, fold):
    n, bits = 1 << 15, 53
    rng = np.random.default_rng(crowd)
    keys = rng.integers(0, 15 << 49, n).astype(np.uint64)
    keys[-crowd - 1:-1] = np.uint64((15 << 49) + 5)  # (in the tile of the last pair, just before it)
    keys[-1] = np.uint64((1 << bits) - 1)
    vals = rng.integers(1, 100, n).astype(np.float64)
    dk, dv = to_dev(keys, torch), to_dev(vals, torch)
    if fold:
        k, v = cuda.sort_reduce(dk, dv, max_key=1 << bits)
        ek, at = np.unique(keys, return_inverse=True)
        ev = np.bincount(at, vals)  # whole numbers: exact in any order
    else:
        k, v = cuda.sort_pairs(dk, dv, max_key=1 << bits)
        ek, ev = oracle.sort_pairs(keys, vals)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0
