"""GPU: the remaindering of the scheme II dense product at the edges of its two
kernels (up to 9, 10 to 16 and more than 16 moduli) and of its 128-row warp
tiles.  Integer operands, on which the scheme is exact: the results are
compared bit for bit."""
import math

import numpy as np
import pytest

from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu

MODULI = (256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193, 191)


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("moduli", range(8, 18))
@pytest.mark.parametrize("h,n,d", [(1, 1, 1), (17, 5, 3), (127, 33, 1), (128, 2, 2), (129, 40, 1), (1100, 300, 1)])
def test_remaindering_exact(cuda, torch, rng, moduli, h, n, d):
    """The last three entries of the inner dimension pair numbers of beta bits
    with zeros, so that the small products next to them stay unscaled: exact
    remainders from -1 and 1 up to the full range."""
    K = 7
    log2m = sum(math.log2(m) for m in MODULI[:moduli])
    beta = min(int(math.floor((log2m - math.log2(K) - 3.0) / 2.0)), 52)
    A = rng.integers(-1, 2, (d, K, h)).astype(np.float64)  # column-major h x K per tab
    B = rng.integers(-1, 2, (d, n, K)).astype(np.float64)
    big = 2.0 ** (beta - 2)  # largest magnitude with scale 1: scaled values stay below 2^(beta - 1)
    A[:, 4, :], B[:, :, 4] = big, 0.0  # scales every row of A and column of B
    A[:, 5, :], B[:, :, 5] = 0.0, big
    A[:, 6, :] = rng.choice([0.0, 0.0, 1.0, -1.0, 3.0, -big], (d, h))
    B[:, :, 6] = rng.choice([0.0, 1.0, -1.0], (d, n))
    ref = np.matmul(B, A)  # sums of at most 5 terms below 2^52: exact
    got = to_host(cuda.dense_mult_crt(to_dev(A.reshape(-1), torch), to_dev(B.reshape(-1), torch), h, K, n, d,
                                      moduli=moduli))
    np.testing.assert_array_equal(got.reshape(d, n, h), ref)
    big = 2.0 ** (min(beta, 26) - 1)
    A = rng.integers(-int(big), int(big), (d, K, h)).astype(np.float64)
    B = rng.integers(-int(big), int(big), (d, n, K)).astype(np.float64)
    got = to_host(cuda.dense_mult_crt(to_dev(A.reshape(-1), torch), to_dev(B.reshape(-1), torch), h, K, n, d,
                                      moduli=moduli))
    ref = np.einsum("dnk,dkh->dnh", B.astype(np.int64), A.astype(np.int64))  # below 2^53: exact
    np.testing.assert_array_equal(got.reshape(d, n, h), ref.astype(np.float64))
    assert cuda.device_status() == 0
