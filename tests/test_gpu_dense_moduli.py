"""GPU: the choice of moduli where an operand holds infinities or NaN.  A row or
column with an infinity has no max / mean ratio (infinity over infinity), and the
call then chooses for a ratio of one, whichever operand it is in; a row with a NaN
has no sum and is left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


@pytest.mark.parametrize("d", [1, 3])
def test_moduli_with_infinities_and_nan(cuda, torch, d):
    import libnt_b200 as L
    h, w, wB = 70, 300, 40
    rng = np.random.default_rng(d)
    A = rng.uniform(0.5, 1, (d, w, h))  # column-major h x w per tab
    B = rng.uniform(0.5, 1, (d, wB, w))
    A[0, 5, 7] = 1e6  # one row's ratio is about 300

    def moduli(a, b):
        return L.dense_crt_moduli(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), h, w, wB, d, 1e-12)

    spread, flat = moduli(A, B), moduli(np.where(A > 1, 1.0, A), B)
    assert spread > flat
    for which, at in ((0, (d - 1, 2, 60)), (0, (0, 2, 7)), (1, (d - 1, 30, 9))):
        ops = [A.copy(), B.copy()]
        ops[which][at] = np.inf
        assert moduli(*ops) == flat
    ops = [A.copy(), B.copy()]
    ops[0][d - 1, 2, 60] = np.nan
    ops[1][0, 3, 4] = np.nan
    assert moduli(*ops) == spread
