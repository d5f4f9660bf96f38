"""GPU: sorts behind a closed gate (95% of the keys in 1/4096 of the range, so
that a bucket overflows) with a poll budget of a few polls.  The queue's waits
between its steps, and its look-backs, then run out; the call latches the sort
look-back bit, or else is right."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu

SORT_LOOKBACK_BIT = 1 << 0


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.fixture
def default_budget(cuda):
    cuda.device_status(clear=True)
    yield
    cuda.set_spin_limit(0)
    cuda.device_status(clear=True)


def _clustered(n, bits, seed=5):
    rng = np.random.default_rng(seed)
    k = rng.integers(0, 1 << bits, n, dtype=np.uint64)
    return np.where(rng.random(n) < 0.95, k >> np.uint64(12), k), rng.uniform(-1, 1, n)


@pytest.mark.parametrize("budget", [1, 100, 2000])
def test_gated_sort_with_a_short_budget(cuda, torch, default_budget, budget):
    n = 1 << 20  # 256 tiles of each of five passes, 444 CTAs
    keys, vals = _clustered(n, 36)
    ek, ev = oracle.sort_pairs(keys, vals)
    dk, dv = to_dev(keys, torch), to_dev(vals, torch)
    cuda.set_spin_limit(budget)
    for _ in range(3):
        k, v = cuda.sort_pairs(dk, dv, max_key=1 << 36)
        word = cuda.device_status(clear=True)
        assert not (word & ~SORT_LOOKBACK_BIT)
        if not word:
            np.testing.assert_array_equal(to_host(k, np.uint64), ek)
            np.testing.assert_array_equal(to_host(v), ev)
    cuda.set_spin_limit(0)
    k, v = cuda.sort_pairs(dk, dv, max_key=1 << 36)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0
