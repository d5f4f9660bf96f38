"""GPU: the expand-sort-compress product with a one-poll budget.  The scan of the
product counts (26 tiles of B entries) may give up on a predecessor and leave a
prefix that does not ascend: the call then latches a look-back bit and stays
inside its buffers, or else is right."""
import numpy as np
import pytest

import oracle
from conftest import rel_ok
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("used", [300, 20])
def test_expand_with_one_poll(cuda, torch, monkeypatch, default_budget, used):
    monkeypatch.setenv("LNT_SPGEMM_ENGINE", "esc")
    h, w, wB, nb = 3000, 300, 250, 60000
    rng = np.random.default_rng(used)
    cols = rng.choice(w, used, replace=False).astype(np.uint64)
    ak = np.unique(rng.integers(0, h, 4000).astype(np.uint64) + np.uint64(h) * cols[rng.integers(0, used, 4000)])
    bk = np.unique(rng.integers(0, w * wB, nb).astype(np.uint64))
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    ek, ev, ea = oracle.lattice_mult(ak, av, h, w, 1, bk, bv, wB, with_abs=True)
    dev = [to_dev(x, torch) for x in (ak, av, bk, bv)]

    def right():
        k, v, _ = cuda.lattice_mult(*dev, h, w, wB, 1)
        return np.array_equal(to_host(k, np.uint64), ek) and rel_ok(to_host(v), ev, ea)

    cuda.set_spin_limit(1)
    for _ in range(5):
        ok = right()
        assert cuda.device_status(clear=True) or ok
    cuda.set_spin_limit(0)
    assert right() and cuda.device_status() == 0
