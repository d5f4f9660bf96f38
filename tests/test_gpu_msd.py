"""GPU: the bucketed sort (partition passes + one CTA per bucket) against the
oracle, at the sizes and key distributions where it can go wrong: one and two
partition passes, tile remainders, either bucket geometry, words that lose
their top key bits, repeated keys inside and beyond a sub-bucket, key-ordered
input, and keys concentrated on the top of the key range.  Every path
restores the input order of equal keys."""
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

# (pairs, max_key): 1 or 2 passes, odd remainders, non-power-of-two ranges
SIZES = [(1 << 20, 1 << 36), ((1 << 20) + 4097, 3 * 10 ** 6), (3 * 10 ** 6 + 1, 7 * 10 ** 8), (1 << 22, 1 << 50),
         (1500001, (1 << 51) + 12345)]


def _keys(rng, n, max_key, kind):
    if kind == "uniform":
        return rng.integers(0, max_key, n, dtype=np.uint64)
    if kind == "sorted":
        return np.sort(rng.integers(0, max_key, n, dtype=np.uint64))
    if kind == "repeated":  # up to a few hundred of a key, never more than a bucket holds
        k = rng.integers(0, max_key, n // 100, dtype=np.uint64)
        return k[rng.integers(0, k.size, n)]
    # the upper half of the range only: buckets twice as full as uniform ones
    return rng.integers(max_key // 2, max_key, n, dtype=np.uint64)


@pytest.mark.parametrize("kind", ["uniform", "sorted", "repeated", "upper"])
@pytest.mark.parametrize("n,max_key", SIZES)
def test_sort_reduce_bucketed(cuda, torch, n, max_key, kind):
    rng = np.random.default_rng(n + len(kind))
    keys = _keys(rng, n, max_key, kind)
    vals = rng.uniform(-1, 1, n)
    vals[rng.random(n) < 0.2] = 0.0
    cut = n // 3
    k, v = cuda.sort_reduce(to_dev(keys[:cut], torch), to_dev(vals[:cut], torch), to_dev(keys[cut:], torch),
                            to_dev(vals[cut:], torch), max_key=max_key, b_scale=-1.0)
    signed = np.concatenate([vals[:cut], -vals[cut:]])
    sk, sv = oracle.sort_pairs(keys, signed)
    ek, ev, ea = oracle.collect_duplicates(sk, sv, with_abs=True)
    np.testing.assert_array_equal(to_host(k, np.uint64), ek)
    # runs are added in input order; only where a bucket overflowed and the
    # general path ran are runs added tile by tile
    assert rel_ok(to_host(v), ev, ea)
    assert cuda.device_status() == 0


# (pairs, max_key): the smallest size taken and its neighbours, one bucket's
# worth, an even and an odd number of digit passes behind the gate, a key so
# wide that the first partition pass takes eight bits
SORTS = [(2047, 1 << 20), (2048, 1 << 20), (2049, 1 << 36), (5121, 1 << 12), (70001, 1 << 40), ((1 << 20) + 3, 1 << 50),
         (600000, 1 << 63)]


@pytest.mark.parametrize("inplace", [False, True])
@pytest.mark.parametrize("kind", ["uniform", "sorted", "one_key", "high_bits"])
@pytest.mark.parametrize("n,max_key", SORTS)
def test_sort_pairs_bucketed(cuda, torch, n, max_key, kind, inplace):
    """Stable and exact whichever path ends up doing it: the bucketed one, or
    (nearly all pairs on one key; keys with bits above the sorted ones, which
    keep them) the gated digit passes behind it."""
    rng = np.random.default_rng(n)
    keys = _keys(rng, n, max_key, "sorted" if kind == "sorted" else "uniform")
    if kind == "one_key":
        keys[rng.random(n) < 0.95] = keys[0]
    vals = rng.uniform(-1, 1, n)
    low = keys.copy()
    if kind == "high_bits" and max_key < 1 << 60:
        keys[::3] |= np.uint64(1 << 61)
    k, v = to_dev(keys, torch), to_dev(vals, torch)
    out = (k, v) if inplace else (None, None)
    k, v = cuda.sort_pairs(k, v, max_key=max_key, out_keys=out[0], out_vals=out[1])
    at = np.argsort(low, kind="stable")
    np.testing.assert_array_equal(to_host(k, np.uint64), keys[at])
    np.testing.assert_array_equal(to_host(v), vals[at])
    assert cuda.device_status() == 0


# extents whose products lie on either side of the limits of the 32-bit and
# the double-precision re-key: 2^31, 2^52, a mode of 2^31 and more
@pytest.mark.parametrize("dims", [[1291, 1291, 1289], [1291, 1290, 1290], [46341, 46341], [1, 2147483647, 1],
                                  [2147483647, 2097151], [2147483648, 3, 5], [67108859, 67108859], [94906265, 94906265],
                                  [7, 11, 13, 17, 19, 23, 29, 31, 37], [3, 5, 1 << 40]])
def test_rekeyed_sort_limits(cuda, torch, dims):
    import libnt_b200 as L
    rng = np.random.default_rng(len(dims))
    total = int(np.prod([int(d) for d in dims], dtype=object))
    n = 6001
    keys = rng.integers(0, total, n, dtype=np.uint64)
    keys[:3] = 0, total - 1, total // 2
    # keys at a mode's boundaries: quotients with remainders 0 and d - 1
    keys[3:1000] = np.minimum(keys[3:1000] // np.uint64(dims[0]) * np.uint64(dims[0]), np.uint64(total - 1))
    keys[1000:2000] = np.minimum(keys[1000:2000] // np.uint64(dims[0]) * np.uint64(dims[0]) + np.uint64(dims[0] - 1),
                                 np.uint64(total - 1))
    vals = rng.uniform(-1, 1, n)
    order = list(range(len(dims)))
    spec = L.RekeySpec.make(dims, order, order[::-1])
    k, v = cuda.permute_sort(to_dev(keys, torch), to_dev(vals, torch), max_key=total, rekey=spec)
    want = oracle.rekey(keys, dims, order, order[::-1])
    at = np.argsort(want, kind="stable")
    np.testing.assert_array_equal(to_host(k, np.uint64), want[at])
    np.testing.assert_array_equal(to_host(v), vals[at])
    assert cuda.device_status() == 0


# one cluster of 1, 2, 4, 8 CTAs, and the first size beyond it
@pytest.mark.parametrize("kind", ["uniform", "sorted", "upper", "one_key", "repeated"])
@pytest.mark.parametrize("max_key", [7, 5000, 3 * 10 ** 6, (1 << 49) - 5])
@pytest.mark.parametrize("n", [1, 33, 2560, 2561, 5121, 10241, 20479, 20480, 20481])
def test_small_sorts(cuda, torch, n, max_key, kind):
    rng = np.random.default_rng(n + max_key % 1000)
    keys = _keys(rng, n, max_key, kind if kind in ("sorted", "upper") else "uniform")
    if kind == "one_key":
        keys[rng.random(n) < 0.9] = keys[0]
    if kind == "repeated":
        keys = keys[rng.integers(0, max(1, n // 3), n)]
    vals = rng.uniform(-1, 1, n)
    vals[rng.random(n) < 0.3] = 0.0
    k, v = cuda.sort_pairs(to_dev(keys, torch), to_dev(vals, torch), max_key=max_key)
    at = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(to_host(k, np.uint64), keys[at])
    np.testing.assert_array_equal(to_host(v), vals[at])
    for skip in (True, False):
        k, v = cuda.sort_reduce(to_dev(keys[: n // 2], torch), to_dev(vals[: n // 2], torch),
                                to_dev(keys[n // 2:], torch), to_dev(vals[n // 2:], torch), max_key=max_key,
                                skip_zero_heads=skip)
        ek, ev, ea = oracle.collect_duplicates(keys[at], vals[at], skip_zero_heads=skip, with_abs=True)
        np.testing.assert_array_equal(to_host(k, np.uint64), ek)
        assert rel_ok(to_host(v), ev, ea)
    assert cuda.device_status() == 0


@pytest.mark.parametrize("entry", ["lnt_sort_pairs", "lnt_permute_sort"])
@pytest.mark.parametrize("n,bits", [(40000, 36), (1 << 20, 20), ((1 << 21) + 3, 36)])
def test_scratch_of_the_digit_passes_is_enough(cuda, torch, rng, monkeypatch, entry, n, bits):
    """With room for the digit passes but not for the bucketed path the sort
    takes the digit passes; with less it is refused."""
    import ctypes as C
    import libnt_b200 as L
    need, have = C.c_size_t(0), C.c_size_t(0)
    query = getattr(L.lib(), entry + "_workspace")
    monkeypatch.setenv("LNT_NO_BUCKETS", "1")
    assert query(n, 1 << bits, C.byref(need)) == 0
    monkeypatch.delenv("LNT_NO_BUCKETS")
    assert query(n, 1 << bits, C.byref(have)) == 0
    keys = rng.integers(0, 1 << bits, n).astype(np.uint64)
    vals = rng.uniform(-1, 1, n)
    k, v = to_dev(keys, torch), to_dev(vals, torch)
    ok, ov = torch.empty_like(k), torch.empty_like(v)
    ws = L.workspace(max(need.value, have.value))

    def call(nbytes):
        p = [C.c_void_p(x.data_ptr()) for x in (k, v, ok, ov, ws)]
        if entry == "lnt_sort_pairs":
            return L.lib().lnt_sort_pairs(p[0], p[1], p[2], p[3], n, 1 << bits, p[4], nbytes, None)
        return L.lib().lnt_permute_sort(p[0], p[1], n, None, p[2], p[3], 1 << bits, p[4], nbytes, None)

    order = np.argsort(keys, kind="stable")
    for nbytes in (need.value, have.value):
        ok.zero_(), ov.zero_()
        assert call(nbytes) == 0
        torch.cuda.synchronize()
        np.testing.assert_array_equal(to_host(ok, np.uint64), keys[order])
        np.testing.assert_array_equal(to_host(ov), vals[order])
    assert call(min(need.value, have.value) - 1) == 5  # LNT_WORKSPACE
    assert cuda.device_status() == 0


@pytest.mark.parametrize("engine", ["esc", "tile"])
def test_products_with_the_scratch_of_the_digit_passes(cuda, torch, rng, monkeypatch, engine):
    """The lattice product's engines likewise: the same C from either scratch."""
    import ctypes as C
    import libnt_b200 as L
    h, w, wB, d = 1500, 60, 40, 2
    ak = np.sort(rng.choice(h * w * d, 60000, replace=False)).astype(np.uint64)
    bk = np.sort(rng.choice(w * wB * d, 1500, replace=False)).astype(np.uint64)
    av, bv = rng.uniform(-1, 1, ak.size), rng.uniform(-1, 1, bk.size)
    da, dav, db, dbv = (to_dev(x, torch) for x in (ak, av, bk, bv))
    monkeypatch.setenv("LNT_SPGEMM_ENGINE", engine)
    A, B = L.Lattice.of(da, dav, h, w, d), L.Lattice.of(db, dbv, w, wB, d)
    n = C.c_size_t(0)
    assert L.lib().lnt_lattice_mult_plan_workspace(C.byref(A), C.byref(B), C.byref(n)) == 0
    plan = L.workspace(n.value)
    counts = torch.empty(2, dtype=torch.int64, device="cuda")
    assert L.lib().lnt_lattice_mult_plan(C.byref(A), C.byref(B), C.c_void_p(plan.data_ptr()), plan.numel(),
                                         C.c_void_p(counts.data_ptr()), None) == 0
    torch.cuda.synchronize()
    products, cap = (int(x) for x in counts.tolist())
    monkeypatch.setenv("LNT_NO_BUCKETS", "1")
    need = C.c_size_t(0)
    assert L.lib().lnt_lattice_mult_workspace(C.byref(A), C.byref(B), products, C.byref(need)) == 0
    monkeypatch.delenv("LNT_NO_BUCKETS")
    have = C.c_size_t(0)
    assert L.lib().lnt_lattice_mult_workspace(C.byref(A), C.byref(B), products, C.byref(have)) == 0
    ek, ev, ea = oracle.lattice_mult(ak, av, h, w, d, bk, bv, wB, with_abs=True)
    for nbytes in (need.value, have.value):
        ws = L.workspace(nbytes)
        ck = torch.empty(cap, dtype=torch.int64, device="cuda")
        cv = torch.empty(cap, dtype=torch.float64, device="cuda")
        nc = torch.empty(1, dtype=torch.int64, device="cuda")
        assert L.lib().lnt_lattice_mult(C.byref(A), C.byref(B), C.c_void_p(plan.data_ptr()), products,
                                        C.c_void_p(ws.data_ptr()), nbytes, C.c_void_p(ck.data_ptr()),
                                        C.c_void_p(cv.data_ptr()), C.c_void_p(nc.data_ptr()), None) == 0
        m = int(nc.item())
        np.testing.assert_array_equal(to_host(ck[:m], np.uint64), ek)
        assert rel_ok(to_host(cv[:m]), ev, ea)
    assert cuda.device_status() == 0


def test_sort_reduce_with_the_scratch_of_the_digit_passes(cuda, torch, rng, monkeypatch):
    import ctypes as C
    import libnt_b200 as L
    n, bits = 1 << 20, 36
    keys = rng.integers(0, 1 << bits, n).astype(np.uint64)
    keys[: n // 8] = keys[n // 8: n // 4]
    vals = rng.uniform(-1, 1, n)
    monkeypatch.setenv("LNT_NO_BUCKETS", "1")
    need = L.sort_reduce_workspace(n, 0, 1 << bits)
    monkeypatch.delenv("LNT_NO_BUCKETS")
    k, v = to_dev(keys, torch), to_dev(vals, torch)
    got = []
    for nbytes in (need, max(need, L.sort_reduce_workspace(n, 0, 1 << bits))):
        ws = L.workspace(nbytes)
        ok, ov = torch.empty_like(k), torch.empty_like(v)
        cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
        assert L.lib().lnt_sort_reduce(C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), n, None, None, None, 0, None,
                                       1.0, 1 << bits, 1, C.c_void_p(ok.data_ptr()), C.c_void_p(ov.data_ptr()),
                                       C.c_void_p(cnt.data_ptr()), C.c_void_p(ws.data_ptr()), nbytes, None) == 0
        m = int(cnt.item())
        got.append((to_host(ok[:m], np.uint64), to_host(ov[:m])))
    sk, sv = oracle.sort_pairs(keys, vals)
    ek, ev = oracle.collect_duplicates(sk, sv)[:2]
    for gk, gv in got:
        np.testing.assert_array_equal(gk, ek)
        np.testing.assert_array_equal(gv, ev)
    assert cuda.device_status() == 0
