"""GPU: the scan merge where pairs and repeats fall on tile boundaries (2048
merged elements): operands that match everywhere, so that a boundary separates
an A from its B, and single keys repeated across a boundary."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("repeat", [0, 2, 5])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 2048, 6000])
def test_pairs_on_tile_boundaries(cuda, torch, n, repeat, shift, op):
    rng = np.random.default_rng(n + repeat)
    ak = np.arange(n, dtype=np.uint64) * np.uint64(3)
    bk = ak[shift:].copy()  # shift 1: every A of a tile's end meets a B of the next tile
    for at in (1022, 1023, 1024, 2047):  # runs of a few equal keys round the boundaries
        if repeat and at + repeat < n:
            ak[at:at + repeat] = ak[at]
            bk[at - shift:at - shift + repeat - 1] = ak[at]
    bk.sort()
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    k, v = cuda.merge_sorted(to_dev(ak, torch), to_dev(av, torch), to_dev(bk, torch), to_dev(bv, torch), op=op)
    ek, ev = oracle.merge_sorted(ak, av, bk, bv, op)[:2]
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("n", [1, 767, 768, 769, 1536, 4608, 460000, 2500000])
def test_tiles_of_1536_and_several_per_cta(cuda, torch, n, op):
    """Tiles of 1536 merged elements, taken in turn by persistent CTAs: one tile,
    two, fewer than there are CTAs, one more each, and several.  Runs of equal
    keys at every second boundary, and outputs that shrink from tile to tile."""
    rng = np.random.default_rng(n)
    ak = np.arange(n, dtype=np.uint64) * np.uint64(2)
    for at in range(766, n - 4, 1536):
        ak[at:at + 4] = ak[at]
    bk = np.where(rng.random(n) < np.linspace(0.0, 1.0, n), ak, ak + np.uint64(1))
    bk.sort()
    av, bv = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    k, v = cuda.merge_sorted(to_dev(ak, torch), to_dev(av, torch), to_dev(bk, torch), to_dev(bv, torch), op=op)
    ek, ev = oracle.merge_sorted(ak, av, bk, bv, op)[:2]
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0
