"""GPU: sorts and folds of few distinct keys, whose runs of equal keys are long:
by result, at the lengths where a run is added up by a lane, by a warp over its row
of 32 and over several rows, and by time, which must not grow with the length
of a run (one thread adding up 20,000 pairs takes over a millisecond)."""
import math

import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


def _fold(keys, vals, skip):
    """Keys, exact sums and sums of magnitudes of the runs that are kept."""
    ek, at = np.unique(keys, return_inverse=True)
    order = np.argsort(at, kind="stable")
    cuts = np.cumsum(np.bincount(at))[:-1]
    runs = np.split(vals[order], cuts)
    kept = [i == 0 or not skip or bool(np.any(r != 0.0)) for i, r in enumerate(runs)]
    ev = np.array([math.fsum(r) for r in runs])
    ea = np.array([math.fsum(np.abs(r)) for r in runs])
    return ek[kept], ev[kept], ea[kept]


def _check(cuda, torch, keys, vals, max_key, skip=True):
    k, v = cuda.sort_reduce(to_dev(keys, torch), to_dev(vals, torch), max_key=max_key, skip_zero_heads=skip)
    ek, ev, ea = _fold(keys, vals, skip)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    # a sum of r terms in any order: at most (r - 1) roundings of 2^-53 each
    worst = int(np.bincount(np.unique(keys, return_inverse=True)[1]).max())
    assert np.all(np.abs(to_host(v) - ev) <= worst * 2.0 ** -53 * ea)
    k, v = cuda.sort_pairs(to_dev(keys, torch), to_dev(vals, torch), max_key=max_key)
    ek, ev = oracle.sort_pairs(keys, vals)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("bits", [12, 30, 49])
@pytest.mark.parametrize("run", [8, 9, 31, 33, 47, 49, 64, 100, 1023, 4000, 20480])
@pytest.mark.parametrize("n", [2000, 20480, 40000])
def test_long_runs(cuda, torch, n, run, bits):
    """n pairs of about n / run keys spread over 2^bits: one cluster, and buckets
    (crowded, or behind a closed gate when they overflow)."""
    rng = np.random.default_rng(n + run)
    kinds = rng.integers(0, 1 << bits, max(1, n // run)).astype(np.uint64)
    keys = kinds[rng.integers(0, kinds.size, n)]
    vals = rng.uniform(-1, 1, n)
    vals[np.isin(keys, kinds[::3])] = 0.0  # runs of zeros only, which are dropped
    _check(cuda, torch, keys, vals, 1 << bits)


@pytest.mark.parametrize("skip", [True, False])
@pytest.mark.parametrize("lengths", [(1, 31, 32, 33, 64, 65, 1, 95, 96, 97, 31), (4096, 1, 1000, 3, 2000), (2500,)])
def test_runs_at_row_ends(cuda, torch, lengths, skip):
    """Known run lengths one after the other, in one cluster and in crowded buckets."""
    rng = np.random.default_rng(len(lengths))
    for copies, gap in ((1, 1), (1, 1 << 20), (12, 1 << 12)):  # (neighbouring keys; far apart; 40,000 pairs)
        keys = np.concatenate([np.full(r, i * gap, np.uint64) for i, r in enumerate(lengths * copies)])
        spread = rng.integers(0, 1 << 34, 25000 if copies > 1 else 0).astype(np.uint64)
        keys = np.concatenate([keys + np.uint64(1 << 33), spread])
        mix = rng.permutation(keys.size)
        _check(cuda, torch, keys[mix], rng.uniform(-1, 1, keys.size), 1 << 34, skip)


@pytest.mark.parametrize("n,kinds", [(2000, 1), (20000, 1), (20000, 10), (1 << 20, 1 << 15), (1 << 22, 1 << 10)])
def test_time_does_not_grow_with_the_runs(cuda, torch, n, kinds):
    """At most five times the time of distinct keys: the serial form was 17 to 55
    times slower at the first two, and three to six at the last two, where the limit
    is two."""
    import libnt_b200 as L
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    vals = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)

    def time(keys, max_key):
        ok, ov = torch.empty_like(keys), torch.empty_like(vals)
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
        ws = L.workspace(L.sort_reduce_workspace(n, 0, max_key))
        best = math.inf
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            L.sort_reduce(keys, vals, max_key=max_key, out_keys=ok, out_vals=ov, count=count, ws=ws, sync=False)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    few = time(torch.randint(0, kinds, (n,), generator=g, device="cuda"), max(2, kinds))
    distinct = time(torch.randperm(n, generator=g, device="cuda"), n)
    assert few < (5.0 if n < 1 << 20 else 2.0) * distinct
