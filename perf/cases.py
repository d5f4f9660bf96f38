"""Performance cases: the calls that programs make through the package's
public functions, from a contraction of two 10,000-entry tensors, where
latency counts, to merges of 2^27 entries and a 16384^3 dense product.

listed() names the cases, draw(rng) makes further ones of the same ranges,
prepare(case, seed) holds what a program has before the call, run(state) is
one pass through the public functions, work(case) the bytes and operations
that a pass cannot do without, exact(case, seed) the result in plain float64
torch.  Sparse coordinates are distinct and uniform unless a case says
otherwise, values uniform in [-1, 1].  A case draws one set of coordinates;
a seed relabels them (every mode's coordinates shifted cyclically, the same
shift for the same label of both operands), shuffles their order and draws the
values, so that results of different seeds have different keys and the same
sizes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libnt_b200 as L

DEV = "cuda"


def listed():
    return [
        # c(i,l) = a(i,j,k) * b(k,l,j) on two small order-3 tensors, the whole
        # index-label product (both operands sorted, then the lattice
        # product): launches and host work count.
        {"name": "contract_small", "kind": "contract", "i": 100, "j": 100, "k": 100, "l": 100, "na": 10000,
         "nb": 10000},
        # the same product with a tall, sparse result (more rows than a
        # column accumulator holds): expand, sort, fold.
        {"name": "contract_tall", "kind": "contract", "i": 5000, "j": 300, "k": 210, "l": 4100, "na": 1100000,
         "nb": 1000000},
        # c(i,j,m) = a(i,j,k,l) * b(k,l,m) with Zipf-distributed contracted
        # coordinates and a dense result, on key-sorted lattices.
        {"name": "contract_skewed", "kind": "skewed", "i": 256, "j": 256, "k": 64, "l": 64, "m": 1024,
         "na": 1 << 21, "nb": 1 << 20},
        # 4096 independent uneven contractions of unsorted tensors in one call.
        {"name": "batch_4096", "kind": "batch", "count": 4096, "dmin": 16, "dmax": 512, "nmin": 100, "nmax": 100000},
        # c = a(i,j,k) + b(k,j,i), small operands, both unsorted.
        {"name": "merge_small", "kind": "merge", "dims": "100x100x100", "na": 10000, "nb": 10000, "op": "+"},
        # an uneven difference of mid-size tensors, extents not powers of two.
        {"name": "merge_ragged", "kind": "merge", "dims": "300x200x150x48", "na": 3100000, "nb": 1700001, "op": "-"},
        # the full-size merge c(i,j,k,l) = a(i,j,k,l) + b(l,k,j,i).
        {"name": "merge_full", "kind": "merge", "dims": "512x512x512x512", "na": 1 << 26, "nb": 1 << 26, "op": "+"},
        # both operands sorted, a under another mode order: re-sort a, merge.
        {"name": "scan_merge", "kind": "scan", "dims": "400x300x500x200", "na": 20000003, "nb": 12000000, "op": "+"},
        # a dense product with an element-wise mode and one operand's modes
        # out of order (permuted copy, choice of moduli, product).
        {"name": "dense_small", "kind": "dense", "h": 300, "w": 260, "n": 220, "d": 3, "permute": True,
         "spread": False},
        # the full-size dense product of the headline, 16384^3 on FP64 operands.
        {"name": "dense_full", "kind": "dense", "h": 16384, "w": 16384, "n": 16384, "d": 1, "permute": False,
         "spread": False},
        # dense times sparse: c(i,l) = A(i,j) * s(j,l).
        {"name": "mixed", "kind": "mixed", "rows": 8192, "cols": 16384, "tabs": 1, "nnz": 1 << 21, "other": 2048,
         "dense_first": True},
        # b(k) = a(i,i,k): a repeated label inside one operand.
        {"name": "unary", "kind": "unary", "n0": 1024, "rest": 65536, "nnz": 1 << 26},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["contract", "tall", "skewed", "batch", "merge", "merge", "scan", "dense", "mixed", "unary"])
    if kind == "contract":
        ext = [rng.randint(20, 300) for _ in range(4)]
        room = min(ext[0], ext[3]) * ext[1] * ext[2] // 4
        n = [min(_log(rng, 500, 300000), room) for _ in range(2)]
        return {"kind": "contract", "i": ext[0], "j": ext[1], "k": ext[2], "l": ext[3], "na": n[0], "nb": n[1]}
    if kind == "tall":
        return {"kind": "contract", "i": _log(rng, 1100, 20000), "j": rng.randint(100, 400), "k": rng.randint(100, 300),
                "l": _log(rng, 500, 8000), "na": _log(rng, 20000, 1200000), "nb": _log(rng, 20000, 1000000)}
    if kind == "skewed":
        return {"kind": "skewed", "i": rng.randint(40, 256), "j": rng.randint(40, 256), "k": rng.randint(20, 64),
                "l": rng.randint(20, 64), "m": rng.randint(300, 1024), "na": _log(rng, 1 << 18, 1 << 21),
                "nb": _log(rng, 1 << 17, 1 << 20)}
    if kind == "batch":
        return {"kind": "batch", "count": _log(rng, 30, 4000), "dmin": 16, "dmax": rng.randint(100, 512), "nmin": 100,
                "nmax": _log(rng, 2000, 100000)}
    if kind in ("merge", "scan"):
        order = rng.randint(2, 5)
        dims = [max(2, int((10 ** rng.uniform(8, 10.8)) ** (1 / order) * rng.uniform(0.5, 1.5))) for _ in range(order)]
        if rng.random() < 0.4:  # small tensors
            dims = [rng.randint(60, 130) for _ in range(3)]
            n = [_log(rng, 1000, 80000) for _ in range(2)]
        else:
            n = [_log(rng, 3000, 30000000) for _ in range(2)]
        return {"kind": kind, "dims": "x".join(map(str, dims)), "na": n[0], "nb": n[1],
                "op": rng.choice(["+", "+", "-"])}
    if kind == "dense":
        return {"kind": "dense", "h": _log(rng, 64, 7000), "w": _log(rng, 64, 7000), "n": _log(rng, 64, 7000),
                "d": rng.choice([1, 1, 2, 5]), "permute": rng.random() < 0.5, "spread": rng.random() < 0.3}
    if kind == "mixed":
        rows, cols = _log(rng, 300, 8000), _log(rng, 300, 8000)
        return {"kind": "mixed", "rows": rows, "cols": cols, "tabs": rng.choice([1, 1, 3]),
                "nnz": min(_log(rng, 3000, 1 << 20), rows * cols // 3), "other": _log(rng, 30, 2048),
                "dense_first": rng.random() < 0.5}
    return {"kind": "unary", "n0": _log(rng, 100, 8000), "rest": _log(rng, 300, 4000), "nnz": _log(rng, 10000, 1 << 25)}


# ---- inputs ---------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _coordinates(total, n, salt):
    """Ascending distinct keys below total (n drawn, repeats collapsed), the same for every seed."""
    return torch.unique(torch.randint(0, total, (n,), generator=_gen(977 + salt), device=DEV))


def _shifts(seed, ext):
    return np.random.default_rng(seed).integers(0, np.asarray(ext)).astype(np.int64)


def _relabel(key, ext, shift):
    """The key (first extent fastest) with every coordinate shifted cyclically;
    extents and shifts are numbers, or one per entry."""
    out, stride = torch.zeros_like(key), 1
    for d, s in zip(ext, shift):
        out += (key % d + s) % d * stride
        key = key // d
        stride = stride * d
    return out


def _shuffled(g, keys):
    return keys[torch.randperm(keys.numel(), generator=g, device=DEV)]


def _values(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * 2 - 1


def _dims(case):
    return [int(x) for x in case["dims"].split("x")]


def _zipf(g, n, dim):
    """Coordinates with P(r) ~ (r + 1)^-1.1."""
    p = torch.arange(1, dim + 1, dtype=torch.float64, device=DEV) ** -1.1
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    return torch.searchsorted(torch.cumsum(p / p.sum(), 0), u).clamp_(max=dim - 1)


def _merge_inputs(case, seed):
    """a unsorted under the mode order 0, 1, ..; b under the reverse order."""
    g = _gen(seed)
    dims = _dims(case)
    total, shift = math.prod(dims), _shifts(seed, dims).tolist()
    ak = _shuffled(g, _relabel(_coordinates(total, case["na"], 0), dims, shift))
    bk = _shuffled(g, _relabel(_coordinates(total, case["nb"], 1), dims[::-1], shift[::-1]))
    return ak, _values(g, ak.numel()), bk, _values(g, bk.numel())


def _contract_inputs(case, seed):
    """a(i,j,k) and b(k,l,j), each unsorted in its own mode order."""
    g = _gen(seed)
    i, j, k, l = (case[x] for x in "ijkl")
    si, sj, sk, sl = _shifts(seed, [i, j, k, l]).tolist()
    ak = _shuffled(g, _relabel(_coordinates(i * j * k, case["na"], 0), (i, j, k), (si, sj, sk)))
    bk = _shuffled(g, _relabel(_coordinates(k * l * j, case["nb"], 1), (k, l, j), (sk, sl, sj)))
    return ak, _values(g, ak.numel()), bk, _values(g, bk.numel())


def _skewed_inputs(case, seed):
    """Key-sorted lattices A (rows (i,j), columns (k,l)) and B (rows (k,l), columns m);
    k and l keep their order of frequency."""
    g, base = _gen(seed), _gen(977)
    na, nb, w = case["na"], case["nb"], case["k"] * case["l"]
    i, j, m = case["i"], case["j"], case["m"]
    si, sj, sm = _shifts(seed, [i, j, m]).tolist()
    row = torch.randint(0, i * j, (na,), generator=base, device=DEV)
    ak = row + i * j * (_zipf(base, na, case["k"]) + case["k"] * _zipf(base, na, case["l"]))
    ak = torch.unique(_relabel(torch.unique(ak), (i, j, w), (si, sj, 0)))
    col = torch.randint(0, m, (nb,), generator=base, device=DEV)
    bk = _zipf(base, nb, case["k"]) + case["k"] * _zipf(base, nb, case["l"]) + w * col
    bk = torch.unique(_relabel(torch.unique(bk), (w, m), (0, sm)))
    av = torch.randn(ak.numel(), generator=g, device=DEV, dtype=torch.float64)
    bv = torch.randn(bk.numel(), generator=g, device=DEV, dtype=torch.float64)
    return ak, av, bk, bv


def _batch_inputs(case, seed):
    """Extents (i, j, k, l) per problem, and the problems' unsorted operands one after another."""
    r, g, base = np.random.default_rng(977), _gen(seed), _gen(977)
    count = case["count"]
    ext = r.integers(case["dmin"], case["dmax"] + 1, (count, 4)).astype(np.int64)
    shift = torch.from_numpy(_shifts(seed, ext)).to(DEV)
    ext_d = torch.from_numpy(ext).to(DEV)
    out = []
    for modes in ((0, 1, 2), (2, 3, 1)):
        size = ext[:, modes].prod(1)
        n = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), count))
        n = np.minimum(np.round(n).astype(np.int64), size // 2 + 1)
        p = torch.repeat_interleave(torch.arange(count, device=DEV), torch.from_numpy(n).to(DEV))
        u = torch.rand(p.numel(), generator=base, device=DEV, dtype=torch.float64)
        key = torch.unique((p << 40) | (u * torch.from_numpy(size).to(DEV)[p]).long())
        p = key >> 40
        off = torch.searchsorted(p, torch.arange(count + 1, device=DEV))
        key = _relabel(key & ((1 << 40) - 1), [ext_d[p, q] for q in modes], [shift[p, q] for q in modes])
        shuffle = torch.argsort((p << 20) | torch.randint(0, 1 << 20, key.shape, generator=g, device=DEV))
        out += [key[shuffle], _values(g, key.numel()), off]
    return ext, out[0], out[1], out[2], out[3], out[4], out[5]


def _dense_inputs(case, seed):
    """Column-major A (h x w x d, or w x h x d where its modes are out of order) and B (w x n x d)."""
    g = _gen(seed)
    h, w, n, d = case["h"], case["w"], case["n"], case["d"]
    x = [_values(g, h * w * d), _values(g, w * n * d)]
    if case["spread"]:  # mantissas times 2^e, e uniform in [-20, 20]
        x = [torch.ldexp(v, torch.randint(-20, 21, v.shape, generator=g, device=DEV)) for v in x]
    return x


def _mixed_inputs(case, seed):
    """The dense operand (other x rows, or cols x other, per tab) and the sparse operand's
    keys, sorted column-major (dense first) or row-major."""
    g = _gen(seed)
    rows, cols, tabs = case["rows"], case["cols"], case["tabs"]
    dense = _values(g, case["other"] * (rows if case["dense_first"] else cols) * tabs)
    ext = (rows, cols, tabs) if case["dense_first"] else (cols, rows, tabs)
    keys = torch.unique(_relabel(_coordinates(rows * cols * tabs, case["nnz"] * tabs, 0), ext, _shifts(seed, ext).tolist()))
    return dense, keys, _values(g, keys.numel())


def _unary_inputs(case, seed):
    """a(i,i',k) sorted under [i, i', k], a tenth of the entries on the diagonal."""
    g = _gen(seed)
    n0, rest = case["n0"], case["rest"]
    keys = _coordinates(n0 * n0 * rest, case["nnz"], 0)
    pick = torch.arange(0, keys.numel(), 10, device=DEV)
    i = keys[pick] % n0
    keys[pick] = i + n0 * i + n0 * n0 * (keys[pick] // (n0 * n0))
    s0, s1 = _shifts(seed, [n0, rest]).tolist()
    keys = torch.unique(_relabel(torch.unique(keys), (n0, n0, rest), (s0, s0, s1)))
    return keys, _values(g, keys.numel())


# ---- the calls --------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("merge", "scan"):
        dims = _dims(case)
        order = list(range(len(dims)))
        st["max_key"] = math.prod(dims)
        ak, av, bk, bv = _merge_inputs(case, seed)
        # both operands are brought to b's order: a's keys are re-keyed
        st["spec"] = L.RekeySpec.make(dims, order, order[::-1])
        st["op"] = 0 if case["op"] == "+" else 1
        na, nb = ak.numel(), bk.numel()
        if kind == "merge":
            st["ws"] = L.workspace(L.sort_reduce_workspace(na, nb, st["max_key"]), DEV)
        else:
            ak, at = torch.sort(ak)
            av = av[at]
            bk, bt = torch.sort(bk)
            bv = bv[bt]
            st["ws"] = L.workspace(L.permute_sort_workspace(na, st["max_key"]), DEV)
            st["sorted"] = (torch.empty_like(ak), torch.empty_like(av))
        st["in"] = (ak, av, bk, bv)
        st["out"] = (torch.empty(na + nb, dtype=torch.int64, device=DEV),
                     torch.empty(na + nb, dtype=torch.float64, device=DEV),
                     torch.zeros(1, dtype=torch.int64, device=DEV))
    elif kind == "contract":
        st["in"] = _contract_inputs(case, seed)
        st["a_key"] = case["i"] * case["j"] * case["k"]
        st["b_key"] = case["k"] * case["l"] * case["j"]
        st["spec_a"] = L.RekeySpec.make([case["i"], case["j"], case["k"]], [0, 1, 2], [0, 1, 2])
        st["spec_b"] = L.RekeySpec.make([case["k"], case["l"], case["j"]], [0, 1, 2], [2, 0, 1])
    elif kind == "skewed":
        st["in"] = _skewed_inputs(case, seed)
    elif kind == "batch":
        ext, ak, av, ao, bk, bv, bo = _batch_inputs(case, seed)
        dims = np.stack([ext[:, 0], ext[:, 1] * ext[:, 2], ext[:, 3], np.ones(len(ext), np.int64)], 1)
        specs = [L.RekeySpec.make([k, l, j], [0, 1, 2], [2, 0, 1]) for _, j, k, l in ext.tolist()]
        st["batch"] = L.Batch(dims, ao.cpu().numpy(), bo.cpu().numpy(), ak, av, bk, bv, a_rekey=[None] * len(ext),
                              b_rekey=specs)
    elif kind == "dense":
        st["in"] = _dense_inputs(case, seed)
        st["out"] = torch.empty(case["h"] * case["n"] * case["d"], dtype=torch.float64, device=DEV)
        st["ws"] = L.workspace(L.dense_crt_workspace(case["h"], case["w"], case["n"], 20), DEV)
    elif kind == "mixed":
        st["in"] = _mixed_inputs(case, seed)
    else:
        st["in"] = _unary_inputs(case, seed)
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "merge":
        ak, av, bk, bv = st["in"]
        ok, ov, cnt = st["out"]
        return L.sort_reduce(ak, av, bk, bv, max_key=st["max_key"], a_rekey=st["spec"],
                             b_scale=-1.0 if st["op"] else 1.0, out_keys=ok, out_vals=ov, count=cnt, ws=st["ws"])
    if kind == "scan":
        ak, av, bk, bv = st["in"]
        ok, ov, cnt = st["out"]
        sk, sv = L.permute_sort(ak, av, max_key=st["max_key"], rekey=st["spec"], out_keys=st["sorted"][0],
                                out_vals=st["sorted"][1], ws=st["ws"])
        return L.merge_sorted(sk, sv, bk, bv, op=st["op"], out_keys=ok, out_vals=ov, count=cnt)
    if kind == "contract":
        ak, av, bk, bv = st["in"]
        sak, sav = L.permute_sort(ak, av, max_key=st["a_key"], rekey=st["spec_a"])
        sbk, sbv = L.permute_sort(bk, bv, max_key=st["b_key"], rekey=st["spec_b"])
        return L.lattice_mult(sak, sav, sbk, sbv, case["i"], case["j"] * case["k"], case["l"])
    if kind == "skewed":
        return L.lattice_mult(*st["in"], case["i"] * case["j"], case["k"] * case["l"], case["m"])
    if kind == "batch":
        b = st["batch"]
        b.run()
        n = int(b.c_off[-1].item())
        return b.c_keys[:n], b.c_vals[:n], b.c_off
    if kind == "dense":
        A, B = st["in"]
        h, w, n, d = case["h"], case["w"], case["n"], case["d"]
        if case["permute"]:
            A = L.dense_permute(A, [w, h, d], [1, 0, 2])
        m = L.dense_crt_moduli(A, B, h, w, n, d)
        return L.dense_mult_crt(A, B, h, w, n, d, moduli=m, out=st["out"], ws=st["ws"])
    if kind == "mixed":
        D, sk, sv = st["in"]
        return L.sparse_dense_mult(D, sk, sv, case["rows"], case["cols"], case["tabs"], case["other"],
                                   case["dense_first"])
    keys, vals = st["in"]
    return L.contract_attract(keys, vals, [case["n0"], case["n0"], case["rest"]], [2], [])


# ---- what a pass cannot do without ------------------------------------------


def _kept(total, n):
    """Expected distinct keys among n uniform draws below total."""
    return -total * math.expm1(-n / total)


def _hit(cells, n):
    """Expected non-empty cells after n uniform hits."""
    return -cells * math.expm1(-n / cells)


def work(case):
    """Operands read once and results written once: 16 B per sparse entry, 8 B per dense one."""
    kind = case["kind"]
    if kind in ("merge", "scan"):
        total = math.prod(_dims(case))
        na, nb = _kept(total, case["na"]), _kept(total, case["nb"])
        out = na + nb - na * nb / total
        return {"bytes": 16 * (na + nb + out), "flops": na * nb / total}
    if kind == "contract":
        con = case["j"] * case["k"]
        na, nb = _kept(case["i"] * con, case["na"]), _kept(case["l"] * con, case["nb"])
        products = na * nb / con
        return {"bytes": 16 * (na + nb + _hit(case["i"] * case["l"], products)), "flops": 2 * products}
    if kind == "skewed":
        p = [np.arange(1, case[x] + 1) ** -1.1 for x in ("k", "l")]
        p = np.outer(p[0] / p[0].sum(), p[1] / p[1].sum())
        h = case["i"] * case["j"]
        a, b = (-c * np.expm1(-n * p / c) for c, n in ((h, case["na"]), (case["m"], case["nb"])))
        products = float((a * b).sum())
        return {"bytes": 16 * (float(a.sum() + b.sum()) + _hit(h * case["m"], products)), "flops": 2 * products}
    if kind == "batch":
        n = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        # E[1 / (j k)] for two uniform extents
        con = (math.log(case["dmax"] / case["dmin"]) / (case["dmax"] - case["dmin"])) ** 2
        products = n * n * con * case["count"]
        return {"bytes": 16 * (2 * n * case["count"] + products), "flops": 2 * products}
    if kind == "dense":
        h, w, n, d = case["h"], case["w"], case["n"], case["d"]
        return {"bytes": 8 * d * (h * w + w * n + h * n), "flops": 2 * d * h * w * n}
    if kind == "mixed":
        rows, cols, tabs, other = case["rows"], case["cols"], case["tabs"], case["other"]
        nnz = _kept(rows * cols * tabs, case["nnz"] * tabs)
        lines, inner = (cols, rows) if case["dense_first"] else (rows, cols)
        out = _hit(lines * tabs, nnz) * other
        return {"bytes": 8 * other * inner * tabs + 16 * (nnz + out), "flops": 2 * nnz * other}
    n = _kept(case["n0"] ** 2 * case["rest"], case["nnz"])
    return {"bytes": 16 * (n + _hit(case["rest"], n / 10)), "flops": n / 10}


# ---- the results in float64 torch ---------------------------------------------


def _reversed_key(key, dims):
    """A key under the mode order 0, 1, .. as a key under the reverse order."""
    out = torch.zeros_like(key)
    for d in dims:
        out = out * d + key % d
        key = key // d
    return out


def _fold(key, val):
    key, at = torch.sort(key, stable=True)
    key, inv = torch.unique_consecutive(key, return_inverse=True)
    return key, torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, inv, val[at])


def _join(acol, arow, av, bcol, blead, bv):
    """Every product of an A and a B entry of one contracted index: (A row, B lead, value)."""
    acol, at = torch.sort(acol)
    lo = torch.searchsorted(acol, bcol)
    n = torch.searchsorted(acol, bcol, right=True) - lo
    e = torch.repeat_interleave(torch.arange(bcol.numel(), device=DEV), n)
    x = at[torch.arange(e.numel(), device=DEV) - (torch.cumsum(n, 0) - n)[e] + lo[e]]
    return arow[x], blead[e], av[x] * bv[e]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("merge", "scan"):
        dims = _dims(case)
        ak, av, bk, bv = _merge_inputs(case, seed)
        if case["op"] == "-":
            bv = -bv
        return _fold(torch.cat([_reversed_key(ak, dims), bk]), torch.cat([av, bv]))
    if kind == "contract":
        ak, av, bk, bv = _contract_inputs(case, seed)
        i, j, k, l = case["i"], case["j"], case["k"], case["l"]
        row, col, val = _join(ak // i, ak % i, av, bk // (k * l) + j * (bk % k), bk // k % l, bv)
        return *_fold(row + i * col, val), val.numel()
    if kind == "skewed":
        ak, av, bk, bv = _skewed_inputs(case, seed)
        h, w, m = case["i"] * case["j"], case["k"] * case["l"], case["m"]
        A = torch.zeros(w * h, dtype=torch.float64, device=DEV)
        A[ak] = av
        B = torch.zeros(m * w, dtype=torch.float64, device=DEV)
        B[bk] = bv
        A, B = A.view(w, h), B.view(m, w)  # column-major: the transposes
        key = torch.nonzero(((B != 0).float() @ (A != 0).float()).view(-1) > 0.5).view(-1)
        products = (torch.bincount(ak // h, minlength=w) * torch.bincount(bk % w, minlength=w)).sum()
        return key, (B @ A).view(-1)[key], int(products.item())
    if kind == "batch":
        ext, ak, av, ao, bk, bv, bo = _batch_inputs(case, seed)
        i, j, k, l = (torch.from_numpy(np.ascontiguousarray(ext[:, q])).to(DEV) for q in range(4))
        problem = torch.arange(len(ext), device=DEV)
        pa, pb = torch.repeat_interleave(problem, ao.diff()), torch.repeat_interleave(problem, bo.diff())
        brow = bk // (k * l)[pb] + j[pb] * (bk % k[pb])
        row, lead, val = _join((pa << 20) | (ak // i[pa]), ak % i[pa], av, (pb << 20) | brow,
                               (pb << 20) | (bk // k[pb] % l[pb]), bv)
        key, val = _fold((lead << 20) | row, val)
        p = key >> 40
        off = torch.searchsorted(p, torch.arange(len(ext) + 1, device=DEV))
        return (key & 0xFFFFF) + i[p] * (key >> 20 & 0xFFFFF), val, off
    if kind == "dense":
        A, B = _dense_inputs(case, seed)
        h, w, n, d = case["h"], case["w"], case["n"], case["d"]
        A = A.view(d, h, w).transpose(1, 2) if case["permute"] else A.view(d, w, h)
        return torch.bmm(B.view(d, n, w), A).reshape(-1)
    if kind == "mixed":
        D, keys, vals = _mixed_inputs(case, seed)
        rows, cols, tabs, other = case["rows"], case["cols"], case["tabs"], case["other"]
        lines, inner = (cols, rows) if case["dense_first"] else (rows, cols)
        S = torch.zeros(tabs * lines * inner, dtype=torch.float64, device=DEV)
        S[keys] = vals
        D = D.view(tabs, inner, other) if case["dense_first"] else D.view(tabs, other, inner).transpose(1, 2)
        full = torch.bmm(S.view(tabs, lines, inner), D).view(tabs * lines, other)
        line = torch.unique_consecutive(keys // inner)
        key = line[:, None] * other + torch.arange(other, device=DEV)
        return key.reshape(-1), full[line].reshape(-1)
    keys, vals = _unary_inputs(case, seed)
    n0 = case["n0"]
    on = keys % n0 == keys // n0 % n0
    key, val = _fold(keys[on] // (n0 * n0), vals[on])
    return key, val, True
