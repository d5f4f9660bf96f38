"""GPU: dense products of several tabs, which run together as far as the
workspace allows: groups of one, of some and of all tabs, odd extents, zero
rows and columns (also next to the padding), and the choice of moduli over all
tabs.  Integer operands: scheme II is exact on them."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_sort import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    return t


def _one_group(h, w, n, moduli, tabs):
    """Workspace bytes of `tabs` tabs: exponents, residues of A, of B and of the products."""
    up, al = (lambda x: (x + 15) // 16 * 16), (lambda x: (x + 255) // 256 * 256)
    M, N, K = up(h), up(n), up(w)
    return al(tabs * h * 4) + al(tabs * n * 4) + sum(al(tabs * moduli * x) for x in (M * K, N * K, M * N))


@pytest.mark.parametrize("tabs_at_once", [1, 2, 16])
@pytest.mark.parametrize("h,w,n,d", [(1, 1, 1, 3), (33, 17, 5, 17), (257, 130, 300, 3), (16, 500, 31, 2)])
def test_tab_groups_exact(cuda, torch, h, w, n, d, tabs_at_once):
    import libnt_b200 as L
    rng = np.random.default_rng(h + n)
    A = rng.integers(-1000, 1001, (d, w, h)).astype(np.float64)  # column-major h x w per tab
    B = rng.integers(-1000, 1001, (d, n, w)).astype(np.float64)
    A[:, :, h // 2] = 0.0   # a zero row of A, a zero column of B
    B[:, n - 1, :] = 0.0
    a, b = to_dev(A.reshape(-1), torch), to_dev(B.reshape(-1), torch)
    ws = L.workspace(_one_group(h, w, n, 14, min(d, tabs_at_once)))
    out = torch.full((h * n * d,), np.nan, dtype=torch.float64, device="cuda")
    st = L.lib().lnt_dense_lattice_mult_crt(*(C.c_void_p(x.data_ptr()) for x in (a, b, out)), h, w, n, d, 14,
                                            C.c_void_p(ws.data_ptr()), ws.numel(), None)
    assert st == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(to_host(out).reshape(d, n, h), np.matmul(B, A))
    # the largest max / mean ratio over all tabs decides, however they are grouped
    m = [L.dense_crt_moduli(a, b, h, w, n, d)]
    small = L.workspace(16 * h + 768)
    got = C.c_int(0)
    assert L.lib().lnt_dense_crt_moduli(C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), h, w, n, d, 1e-12,
                                        C.c_void_p(small.data_ptr()), small.numel(), C.byref(got), None) == 0
    m.append(got.value)
    m.append(max(L.dense_crt_moduli(a[t * h * w:(t + 1) * h * w], b[t * w * n:(t + 1) * w * n], h, w, n)
                 for t in range(d)))
    assert m[0] == m[1] == m[2]
    assert cuda.device_status() == 0
