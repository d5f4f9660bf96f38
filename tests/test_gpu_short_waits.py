"""GPU: calls whose kernels wait for one another's tiles or buckets, with a budget of
one poll: the digit passes, the bucketed fold, the scan merge.  Each call latches
its look-back bit, or else is right; with the default budget it is right."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu

SORT_BIT, REDUCE_BIT, MERGE_BIT = 1 << 0, 1 << 1, 1 << 2


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


def _run(cuda, call, want, bit):
    def right():
        k, v = call()
        return np.array_equal(to_host(k, np.uint64), want[0]) and np.array_equal(to_host(v), want[1])

    cuda.set_spin_limit(1)
    for _ in range(4):
        ok = right()
        word = cuda.device_status(clear=True)
        assert word & ~bit == 0 and (word or ok)
    cuda.set_spin_limit(0)
    assert right() and cuda.device_status() == 0


def test_digit_passes(cuda, torch, monkeypatch, default_budget):
    """2^22 pairs: over a thousand tiles in each of five passes."""
    monkeypatch.setenv("LNT_NO_BUCKETS", "1")
    rng = np.random.default_rng(5)
    keys, vals = rng.integers(0, 1 << 36, 1 << 22, dtype=np.uint64), rng.uniform(-1, 1, 1 << 22)
    dk, dv = to_dev(keys, torch), to_dev(vals, torch)
    _run(cuda, lambda: cuda.sort_pairs(dk, dv, max_key=1 << 36), oracle.sort_pairs(keys, vals), SORT_BIT)


def test_bucketed_fold(cuda, torch, default_budget):
    """2^22 pairs of 2^21 keys in 2^11 buckets, whose offsets come from a look-back."""
    rng = np.random.default_rng(6)
    keys, vals = rng.integers(0, 1 << 21, 1 << 22, dtype=np.uint64), rng.integers(1, 9, 1 << 22).astype(np.float64)
    ek, at = np.unique(keys, return_inverse=True)
    dk, dv = to_dev(keys, torch), to_dev(vals, torch)
    _run(cuda, lambda: cuda.sort_reduce(dk, dv, max_key=1 << 21), (ek, np.bincount(at, vals)), REDUCE_BIT)


def test_scan_merge(cuda, torch, default_budget):
    """2 x 2^21 pairs: 2731 tiles, several per CTA."""
    rng = np.random.default_rng(7)
    ak, bk = (np.unique(rng.integers(0, 1 << 23, 1 << 21, dtype=np.uint64)) for _ in range(2))
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    dev = [to_dev(x, torch) for x in (ak, av, bk, bv)]
    _run(cuda, lambda: cuda.merge_sorted(*dev), oracle.merge_sorted(ak, av, bk, bv, 0)[:2], MERGE_BIT)
