"""GPU: the chunked fold behind contract_attract at its edges: sizes round a
row, a batch, a chunk and a tile, groups of one entry, of a few, of many
chunks, and one group over everything; keys exact, values within 1e-12 *
sum|terms|."""
import numpy as np
import pytest

from conftest import rel_ok
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("n0", [64, 37])
@pytest.mark.parametrize("run", [1, 3, 31, 32, 257, 5000, 10 ** 7])
@pytest.mark.parametrize("n", [1, 31, 33, 256, 257, 2047, 2049, 70001, 1 << 21])
def test_fold_group_lengths(cuda, torch, n, run, n0):
    """b(k) = a(i,i',k): about `run` entries per k (at most n0^2, repeats allowed)."""
    rng = np.random.default_rng(n + run + n0)
    group = np.sort(rng.integers(0, max(1, n // run), n).astype(np.uint64))
    i = rng.integers(0, n0, n).astype(np.uint64)
    j = np.where(rng.random(n) < 0.5, i, rng.integers(0, n0, n).astype(np.uint64))
    keys = np.sort(i + np.uint64(n0) * j + np.uint64(n0 * n0) * group)
    vals = rng.uniform(-1, 1, n)
    rest = int(group.max()) + 1
    k, v, flag = cuda.contract_attract(to_dev(keys, torch), to_dev(vals, torch), [n0, n0, rest], [2], [])
    con = keys % np.uint64(n0 * n0)
    on = con % np.uint64(n0) == con // np.uint64(n0)
    g = (keys // np.uint64(n0 * n0))[on]
    ek, at = np.unique(g, return_inverse=True)
    ev, ea = np.zeros(ek.size), np.zeros(ek.size)
    np.add.at(ev, at, vals[on])
    np.add.at(ea, at, np.abs(vals[on]))
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    assert rel_ok(to_host(v), ev, ea) and flag
    assert cuda.device_status() == 0
