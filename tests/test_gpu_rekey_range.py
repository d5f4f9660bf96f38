"""GPU: keys beyond their tensor's extents in the sorts that re-key on the fly.
The reference's re-key decodes such a key with its last mode's index beyond the
extent; the sorts' 32-bit and double-reciprocal forms have to agree with the
64-bit one (lnt_rekey) on it, wherever they are taken."""
import numpy as np
import pytest

import oracle
from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


# (extents, new order, keys beyond the extents)
CASES = [((1000, 1000, 2000), (1, 0, 2), (4294000999, 4294000000, 4293999999, 2 ** 32 - 1, 2 ** 32, 2 ** 40)),
         ((3, 7, 90000), (1, 0, 2), (2 ** 31, 2 ** 32 - 1, 2 ** 32 - 2, 2 ** 33 + 5)),
         ((3, 10 ** 9), (1, 0), (10 ** 13, 2 ** 45, 2 ** 33, 3 * (2 ** 32 - 1), 3 * (2 ** 32 - 1) - 1, 2 ** 47 - 1)),
         ((5, 4, 10 ** 8 + 7), (1, 0, 2), (2 ** 47 - 1, 20 * (2 ** 32 - 1), 20 * 2 ** 32, 2 ** 34))]


@pytest.mark.parametrize("n", [3000, 30000])
@pytest.mark.parametrize("dims,order,beyond", CASES)
def test_permute_sort_of_keys_beyond_the_extents(cuda, torch, dims, order, beyond, n):
    import libnt_b200 as L
    rng = np.random.default_rng(n)
    total = int(np.prod([int(d) for d in dims], dtype=object))
    keys = rng.integers(0, total, n).astype(np.uint64)
    at = rng.choice(n, len(beyond), replace=False)
    keys[at] = np.array(beyond, np.uint64)
    vals = rng.uniform(-1, 1, n)
    cur = list(range(len(dims)))
    full = to_host(cuda.rekey(to_dev(keys, torch), dims, cur, order), np.uint64)
    for i in range(n) if n < 5000 else at:  # the re-key itself, in whole numbers
        k, digit = int(keys[i]), []
        for d in dims[:-1]:
            k, r = divmod(k, d)
            digit.append(r)
        digit.append(k)
        stride, want = 1, 0
        for m in order:
            want += digit[m] * stride
            stride *= dims[m]
        assert int(full[i]) == want
    k, v = cuda.permute_sort(to_dev(keys, torch), to_dev(vals, torch), max_key=1 << 48,
                             rekey=L.RekeySpec.make(dims, cur, order))
    ek, ev = oracle.sort_pairs(full, vals)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    np.testing.assert_array_equal(to_host(v), ev)
    assert cuda.device_status() == 0
