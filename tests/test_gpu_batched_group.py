"""GPU: the batched contraction of unsorted tensors at its edges: operands of
several tasks and of none, no matching index, several tabs, dense columns
walked by a whole warp, repeated keys, 512 rows (grouped) and 513 (sorted),
lattices whose keys need more than 32 bits.  Keys exact, values within 1e-12 *
sum|terms|."""
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


def _problem(rng, h, w, wB, d, na, nb, repeat=False):
    a = rng.integers(0, h * w * d, na).astype(np.uint64)
    b = rng.integers(0, w * wB * d, nb).astype(np.uint64)
    if not repeat:
        a, b = rng.permutation(np.unique(a)), rng.permutation(np.unique(b))
    return (h, w, wB, d), a, rng.uniform(-1, 1, a.size), b, rng.uniform(-1, 1, b.size)


SETS = {
    "one big": [(300, 5000, 200, 1, 200000, 150000, False)],
    "uneven": [(1, 1, 1, 1, 1, 1, False), (512, 37, 3, 2, 5000, 60, False), (17, 100000, 9, 1, 50, 70000, False),
               (40, 30, 20, 1, 0, 100, False), (40, 30, 20, 1, 100, 0, False), (511, 4, 700, 1, 2000, 2800, False),
               (33, 64, 65, 3, 3000, 3000, True)],
    "no partner": [(100, 10 ** 6, 100, 1, 3, 3, False), (8, 8, 8, 1, 64, 64, False)],
    "wide keys": [(500, 1 << 25, 400, 1, 30000, 30000, False), (512, 9, 1 << 22, 1, 4000, 20000, False)],
    "sorted path": [(513, 50, 40, 1, 5000, 1000, False), (20, 50, 40, 1, 500, 1000, False)],
}


@pytest.mark.parametrize("name", SETS)
def test_batched_contract_edges(cuda, torch, name):
    import libnt_b200 as L
    rng = np.random.default_rng(len(name))
    probs = [_problem(rng, *c) for c in SETS[name]]
    if name == "no partner":  # the first problem's operands share no contracted index
        (h, w, wB, d), a, av, b, bv = probs[0]
        a, b = np.array([5, 205], np.uint64), np.array([3, 9], np.uint64)
        probs[0] = ((h, w, wB, d), a, av[:2], b, bv[:2])
    dims = np.array([p[0] for p in probs], np.int64)
    off = [np.concatenate([[0], np.cumsum([p[i].size for p in probs])]).astype(np.uint64) for i in (1, 3)]
    cat = [to_dev(np.concatenate([p[i] for p in probs]), torch) for i in (1, 2, 3, 4)]
    batch = L.Batch(dims, *off, *cat, a_rekey=[None] * len(probs))
    for _ in range(2):  # the workspace is reused
        batch.run()
    for p, ((h, w, wB, d), a, av, b, bv) in enumerate(probs):
        oa, ob = np.argsort(a, kind="stable"), np.argsort(b, kind="stable")
        ek, ev, ea = oracle.lattice_mult(a[oa], av[oa], h, w, d, b[ob], bv[ob], wB, with_abs=True)
        k, v = batch.result(p)
        np.testing.assert_array_equal(to_host(k, np.uint64), ek)
        assert rel_ok(to_host(v), ev, ea)
    assert cuda.device_status() == 0
