"""GPU: a batch prepared on one stream and run on another.  The prepare call is
synchronous, so nothing orders the two.  One problem has 2^21 output columns:
its part of the column order takes milliseconds to write."""
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


@pytest.mark.parametrize("unsorted", [True, False])
def test_prepare_and_run_on_different_streams(cuda, torch, unsorted):
    import libnt_b200 as L
    rng = np.random.default_rng(3)
    probs = []
    for h, w, wB, na, nb in ((64, 9, 1 << 21, 400, 30000), (40, 300, 50, 2000, 2500)):
        a, b = np.unique(rng.integers(0, h * w, na).astype(np.uint64)), np.unique(
            rng.integers(0, w * wB, nb).astype(np.uint64))
        if unsorted:
            a, b = rng.permutation(a), rng.permutation(b)
        probs.append(((h, w, wB, 1), a, rng.uniform(-1, 1, a.size), b, rng.uniform(-1, 1, b.size)))
    dims = np.array([p[0] for p in probs], np.int64)
    off = [np.concatenate([[0], np.cumsum([p[i].size for p in probs])]).astype(np.uint64) for i in (1, 3)]
    cat = [to_dev(np.concatenate([p[i] for p in probs]), torch) for i in (1, 2, 3, 4)]
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(first):
        batch = L.Batch(dims, *off, *cat, a_rekey=[None] * len(probs) if unsorted else None)
    with torch.cuda.stream(second):
        batch.run()
    torch.cuda.synchronize()
    for p, ((h, w, wB, d), a, av, b, bv) in enumerate(probs):
        oa, ob = np.argsort(a, kind="stable"), np.argsort(b, kind="stable")
        ek, ev, ea = oracle.lattice_mult(a[oa], av[oa], h, w, d, b[ob], bv[ob], wB, with_abs=True)
        k, v = batch.result(p)
        np.testing.assert_array_equal(to_host(k, np.uint64), ek)
        assert rel_ok(to_host(v), ev, ea)
    assert cuda.device_status() == 0
