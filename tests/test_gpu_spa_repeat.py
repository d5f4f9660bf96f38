"""GPU: the accumulator engine adds up in an order that does not depend on the
run: repeated products have the same bits, with a CTA per output column (few
columns) and with a warp per column."""
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


# (rows, contracted, columns, tabs, entries of A, of B)
CASES = [(64, 2000, 100, 1, 30000, 60000), (1000, 500, 40, 2, 100000, 8000), (7, 3000, 9, 1, 15000, 20000),
         (100, 400, 5000, 1, 20000, 300000)]


@pytest.mark.parametrize("h,w,wB,d,na,nb", CASES)
def test_products_repeat_exactly(cuda, torch, h, w, wB, d, na, nb):
    rng = np.random.default_rng(h)
    ak = np.unique(rng.integers(0, h * w * d, na).astype(np.uint64))
    bk = np.unique(rng.integers(0, w * wB * d, nb).astype(np.uint64))
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    dev = [to_dev(x, torch) for x in (ak, av, bk, bv)]
    k, v, _ = cuda.lattice_mult(*dev, h, w, wB, d)
    k, v = to_host(k, np.uint64), to_host(v)
    ek, ev, ea = oracle.lattice_mult(ak, av, h, w, d, bk, bv, wB, with_abs=True)
    np.testing.assert_array_equal(k, ek)
    assert rel_ok(v, ev, ea)
    for _ in range(20):
        v2 = to_host(cuda.lattice_mult(*dev, h, w, wB, d)[1])
        np.testing.assert_array_equal(v2.view(np.int64), v.view(np.int64))
    assert cuda.device_status() == 0
