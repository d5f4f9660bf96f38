"""GPU: the scan merge with pairs and runs of equal keys round its tile ends.  A
tile is 1536 merged elements, so two operands that match everywhere cross one
every 768 keys: runs of a few equal keys begin just before, at and just behind
every such place, in A, in B, or in both."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu

TILE = 1536


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("repeat", [2, 5])
@pytest.mark.parametrize("which", ["a", "b", "both"])
def test_runs_round_tile_ends(cuda, torch, which, repeat, shift, op):
    n = 9 * TILE // 2 + 7
    rng = np.random.default_rng(repeat + 10 * shift)
    for off in (-repeat, -2, -1, 0, 1):
        ak = np.arange(n, dtype=np.uint64) * np.uint64(3)
        bk = ak[shift:].copy()  # (shift 1: B's partner comes one element later)
        for at in range(TILE // 2, n - 2 * repeat, TILE // 2):
            if which != "b":
                ak[at + off:at + off + repeat] = ak[at + off]
            if which != "a":
                bk[at - shift + off:at - shift + off + repeat] = bk[at - shift + off]
        av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
        k, v = cuda.merge_sorted(to_dev(ak, torch), to_dev(av, torch), to_dev(bk, torch), to_dev(bv, torch), op=op)
        ek, ev = oracle.merge_sorted(ak, av, bk, bv, op)[:2]
        np.testing.assert_array_equal(to_host(k, np.uint64), ek)
        np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0
