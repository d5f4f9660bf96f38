"""GPU: contract_attract with a one-poll budget.  Its chunk scan (several tiles)
and its group fold may give up on a predecessor: the call then latches a
look-back bit and stays inside its buffers, or else is right."""
import numpy as np
import pytest

from conftest import rel_ok
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu

LOOKBACK_BITS = (1 << 1) | (1 << 3)  # fold, scan


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


def test_contract_attract_with_one_poll(cuda, torch, default_budget):
    """b(k) = a(i,i',k): 2^22 entries in 16384 chunks, eight tiles of the scan."""
    n, n0 = 1 << 22, 16
    rng = np.random.default_rng(9)
    group = np.sort(rng.integers(0, n // 3, n).astype(np.uint64))
    i = rng.integers(0, n0, n).astype(np.uint64)
    j = np.where(rng.random(n) < 0.5, i, rng.integers(0, n0, n).astype(np.uint64))
    keys = np.sort(i + np.uint64(n0) * j + np.uint64(n0 * n0) * group)
    vals = rng.uniform(-1, 1, n)
    con = keys % np.uint64(n0 * n0)
    on = con % np.uint64(n0) == con // np.uint64(n0)
    ek, at = np.unique((keys // np.uint64(n0 * n0))[on], return_inverse=True)
    ev, ea = np.bincount(at, vals[on]), np.bincount(at, np.abs(vals[on]))
    dk, dv = to_dev(keys, torch), to_dev(vals, torch)
    dims = [n0, n0, int(group.max()) + 1]

    def right():
        k, v, _ = cuda.contract_attract(dk, dv, dims, [2], [])
        return np.array_equal(to_host(k, np.uint64), ek) and rel_ok(to_host(v), ev, ea)

    cuda.set_spin_limit(1)
    for _ in range(5):
        ok = right()
        word = cuda.device_status(clear=True)
        assert word & LOOKBACK_BITS if word else ok
    cuda.set_spin_limit(0)
    assert right() and cuda.device_status() == 0
