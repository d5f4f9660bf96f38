"""GPU: the product expansion of the expand-sort-compress engine at its edges:
product counts round a tile of 2048, B entries without products between those
with (more than a tile decodes at once), single long A columns, several tabs."""
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


# (rows, contracted, columns, tabs, A columns used, B entries)
CASES = [(3000, 50, 40, 1, 50, 60), (2048, 1, 1, 1, 1, 1), (2049, 1, 3, 1, 1, 3), (4000, 5000, 300, 1, 7, 20000),
         (1500, 200, 100, 3, 200, 1000), (20000, 3, 2, 2, 3, 8)]


@pytest.mark.parametrize("h,w,wB,d,used,nb", CASES)
def test_expand_matches_oracle(cuda, torch, monkeypatch, h, w, wB, d, used, nb):
    monkeypatch.setenv("LNT_SPGEMM_ENGINE", "esc")
    rng = np.random.default_rng(h + nb)
    cols = np.concatenate([rng.choice(w, used, replace=False) + w * t for t in range(d)]).astype(np.uint64)
    ak = np.unique(rng.integers(0, h, 40 * h // 10).astype(np.uint64)
                   + np.uint64(h) * cols[rng.integers(0, cols.size, 40 * h // 10)])
    bk = np.unique(rng.integers(0, w * wB * d, nb).astype(np.uint64))
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    k, v, products = cuda.lattice_mult(to_dev(ak, torch), to_dev(av, torch), to_dev(bk, torch), to_dev(bv, torch), h, w,
                                       wB, d)
    ek, ev, ea = oracle.lattice_mult(ak, av, h, w, d, bk, bv, wB, with_abs=True)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    assert rel_ok(to_host(v), ev, ea)
    assert cuda.device_status() == 0
