"""Edges of the kernels that a rule on sizes, types or alignment selects:
each path against the oracle, or against the general path over the same data.

Bar: bit-exact (integers, permutations, and f64 sums against the oracle's
restatement of the fixed summation order).
"""
import ctypes as C
import os

import numpy as np
import pytest

from horsepower_gb300.abi import (Builtins, DTYPE, H_B, H_C, H_E, H_F, H_H, H_I, H_J, H_L)  # noqa: F401

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def libs():
    import subprocess
    import horsepower_gb300
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle"), "port"], check=True)
    ora = Builtins(os.path.join(ROOT, "oracle", "_build", "liboracle.so"), "oracle")
    ora.lib.hgoTreeSumF64.restype = C.c_double
    ora.lib.hgoTreeSumF64.argtypes = [C.c_void_p, C.c_longlong]
    return horsepower_gb300.load(), ora


@pytest.mark.parametrize("sizes", [
    [33, 64, 255, 256, 257, 288, 511, 512],            # a block of segments one warp takes each
    [513, 514, 767, 768, 769, 1024, 4095, 4096],       # a block of segments all warps share
    [33, 513, 34, 4096, 512, 40, 2049, 256, 700] * 9,  # both in one block, and a last block not full
])
def test_mid_size_groups(libs, sizes):
    """Groups of 33 to 4096 rows: sums equal the fixed tile tree of their rows
    bit for bit, min and max equal numpy's, on either side of 512 rows."""
    gpu, ora = libs
    rng = np.random.default_rng(len(sizes))
    key = np.repeat(np.arange(len(sizes), dtype=np.int64) + 70_000 * (np.arange(len(sizes)) % 2), sizes)
    rng.shuffle(key)
    pay = rng.standard_normal(key.size) * 10.0 ** rng.integers(-8, 8, key.size)
    ipay = rng.integers(-2 ** 31, 2 ** 31, key.size).astype(np.int32)
    g = gpu.call("pfnGroup", gpu.vec(key, H_L))
    vals = gpu.call("pfnValues", g)
    keys = gpu.to_py(gpu.call("pfnKeys", g))
    sums = gpu.to_py(gpu.call("hgpuGroupSum", gpu.vec(pay, H_E), vals))
    lo = gpu.to_py(gpu.call("hgpuGroupMin", gpu.vec(ipay, H_I), vals))
    hi = gpu.to_py(gpu.call("hgpuGroupMax", gpu.vec(pay, H_E), vals))
    for gi, first in enumerate(keys):
        rows = np.flatnonzero(key == key[first])
        x = np.ascontiguousarray(pay[rows])
        want = ora.lib.hgoTreeSumF64(x.ctypes.data, x.size)
        assert sums[gi].tobytes() == np.float64(want).tobytes(), (len(rows), sums[gi], want)
        assert lo[gi] == ipay[rows].min() and hi[gi] == x.max()
    gpu.free_inputs()


def key_column(rng, n, lo_bit, hi_bit, negative=False):
    """n i64 keys whose varying bits are lo_bit .. hi_bit - 1 (repeats included)."""
    top = rng.integers(0, 1 << min(hi_bit - lo_bit, 62), n, dtype=np.int64)
    top[rng.random(n) < 0.2] = top[0]
    top[:2] = [0, (1 << (hi_bit - lo_bit)) - 1]
    key = top << lo_bit
    return -key if negative else key


@pytest.mark.parametrize("n", [2, 31, 4095, 4096, 4097, 70_001, 2_000_003])
@pytest.mark.parametrize("lo_bit,hi_bit", [(0, 1), (0, 8), (0, 9), (0, 17), (3, 20), (0, 32), (0, 33), (5, 45), (0, 45),
                                           (0, 53), (0, 62)])
def test_radix_keys(libs, n, lo_bit, hi_bit):
    """@order and @group of one i64 key for key widths on either side of what
    a 64-bit record holds beside the row id (whole, without the first digit,
    not at all), constant low bits, and tile and chunk remainders: the stable
    argsort, its reverse when descending, and its runs."""
    gpu = libs[0]
    rng = np.random.default_rng(n + 100 * hi_bit + lo_bit)
    key = key_column(rng, n, lo_bit, hi_bit)
    want = np.argsort(key, kind="stable")
    k = gpu.vec(key, H_L)
    up = gpu.to_py(gpu.call("pfnOrderBy", k, gpu.vec(np.array([1], bool), H_B)))
    assert np.array_equal(up, want)
    down = gpu.to_py(gpu.call("pfnOrderBy", k, gpu.vec(np.array([0], bool), H_B)))
    assert np.array_equal(down, want[::-1])
    if n > 100_000 and hi_bit > 20:
        gpu.free_inputs()
        return  # a million one-row groups say no more than the small sizes
    g = gpu.to_py(gpu.call("pfnGroup", k))
    heads = np.flatnonzero(np.r_[True, key[want][1:] != key[want][:-1]])
    assert np.array_equal(g[1], want[heads])
    assert np.array_equal(np.concatenate(g[2]), want)
    assert [len(v) for v in g[2]] == list(np.diff(np.r_[heads, n]))
    gpu.free_inputs()


@pytest.mark.parametrize("t0,t1", [(H_I, H_I), (H_L, H_I), (H_I, H_L), (H_L, H_L)])
@pytest.mark.parametrize("dirs", [(1, 1), (0, 1), (1, 0), (0, 0)])
@pytest.mark.parametrize("span0,span1", [(1 << 8, 1 << 8), (1 << 16, 1 << 18), (1 << 29, 1 << 16), (1 << 30, 1 << 30)])
def test_radix_pairs(libs, t0, t1, dirs, span0, span1):
    """@order of two integer columns of every width and direction, packed keys
    of 16 to 60 bits, negative values included: the oracle's permutation."""
    gpu, ora = libs
    rng = np.random.default_rng(span0 % 97 + 7 * dirs[0] + dirs[1])
    n = 40_009
    a = (rng.integers(0, span0, n) - span0 // 2).astype(np.int32 if t0 == H_I else np.int64)
    b = (rng.integers(0, span1, n) - span1 // 3).astype(np.int32 if t1 == H_I else np.int64)
    a[: n // 2] = a[rng.integers(0, 50, n // 2)]
    out = []
    for L in (gpu, ora):
        z = L.call("pfnOrderBy", L.list([L.vec(a, t0), L.vec(b, t1)]), L.vec(np.array(dirs, bool), H_B))
        out.append(L.to_py(z))
        L.free_inputs()
    assert np.array_equal(out[0], out[1])


def quick_keys(rng, n, shape):
    x = rng.standard_normal(n)
    if shape == "ties":
        x = np.round(x * 3) / 2
    elif shape == "few":
        x = rng.integers(0, 3, n) * 0.5
    elif shape == "equal":
        x = np.full(n, -0.0)
        x[::3] = 0.0
    elif shape == "rising":  # first-element pivots: one element per depth
        x = np.sort(x)
        x[: n // 3] = x[0]
    elif shape == "falling":
        x = np.sort(x)[::-1].copy()
    return x


@pytest.mark.parametrize("shape", ["plain", "ties", "few", "equal", "rising", "falling"])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 64, 65, 1000, 4095, 4096, 4097, 4200, 9000])
def test_quicksort_scales(libs, n, shape):
    """The quicksort in a warp, in a CTA and in global memory: f64 keys on
    either side of 32 and 4096 rows, both directions, against the oracle's
    sequential quicksort (its order of equal keys included)."""
    gpu, ora = libs
    x = quick_keys(np.random.default_rng(n), n, shape)
    for up in (1, 0):
        out = []
        for L in (gpu, ora):
            out.append(L.to_py(L.call("pfnOrderBy", L.vec(x, H_E), L.vec(np.array([up], bool), H_B))))
            L.free_inputs()
        assert np.array_equal(out[0], out[1]), up


@pytest.mark.parametrize("dirs", [(1, 1), (0, 1), (1, 0), (0, 0)])
@pytest.mark.parametrize("second", ["i32", "f64", "char"])
@pytest.mark.parametrize("run", [1, 2, 9, 10, 32, 33, 700, 5000])
def test_quicksort_lists(libs, run, second, dirs):
    """Lists led by an f64 column whose runs of equal values have about `run`
    rows: short runs only (sorted by a warp each), longer ones, and no repeats
    at all, with a stable, a quicksort and a char column behind it."""
    gpu, ora = libs
    if second == "char" and not dirs[1]:
        pytest.skip("descending char columns are refused")
    rng = np.random.default_rng(run + 3 * dirs[0] + dirs[1])
    n = 12_007
    a = rng.permutation(n) // run * 0.25
    b = {"i32": (rng.integers(-4, 4, n).astype(np.int32), H_I), "f64": (rng.integers(-4, 4, n) * 1.5, H_E),
         "char": (rng.integers(97, 103, n).astype(np.int8), H_C)}[second]
    out = []
    for L in (gpu, ora):
        z = L.call("pfnOrderBy", L.list([L.vec(a, H_E), L.vec(*b)]), L.vec(np.array(dirs, bool), H_B))
        out.append(L.to_py(z))
        L.free_inputs()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("nfact,groups", [(2047, 6), (2048, 8), (2049, 1), (100_003, 6), (300_001, 8)])
def test_shared_windows(libs, nfact, groups):
    """Plans over one table set, date windows from none to all of the rows (a
    tile's selection fits one list, or is taken in parts): each plan's rows
    equal the same plan through its builtins, bit for bit."""
    from horsepower_gb300 import batch as B, data as D, plans as P
    gpu = libs[0]
    dim, fact = D.join_tables(nfact=nfact, ndim=max(2, nfact // 3), seed=nfact)
    rng = np.random.default_rng(groups)
    g = rng.integers(0, groups, nfact)
    fact["flag"], fact["status"] = (g // 2).astype(np.int8), (g % 2).astype(np.int8)
    ddim, dfact = B.device_tables(gpu, dim, fact)
    spans = [1, 30, 365, 620, 640, 700, 1300, 2525, 2526]
    wins = [(D.DAYS0 + int(rng.integers(0, D.NDAYS - s + 1)), s) for s in spans]
    wins = [(lo, lo + s) for lo, s in wins] + [(D.WIN_LO, D.WIN_LO), (D.DAYS0 - 9, D.DAYS0 + 5000)]
    got = B.run_batch(gpu, [B.make_plan(ddim, dfact, lo, hi) for lo, hi in wins])
    for (lo, hi), r in zip(wins, got):
        if not np.isin(fact["fk"], dim["pk"][(dim["date"] >= lo) & (dim["date"] < hi)]).any():
            assert len(r[0]) == 0
            continue
        want = [gpu.to_py(o) for o in P.join_group(gpu, ddim, dfact, lo, hi)]
        for a, b in zip(r, want):
            assert np.array_equal(a, b), (lo, hi)
    gpu.free_inputs()


@pytest.mark.parametrize("nreq", [1, 7, 8, 9, 40])
def test_served_windows(libs, nreq):
    """Served filter-aggregates, any number of windows folded together: each
    equals the fused chain of its window bit for bit.  Served top-k rows equal
    the first rows of the stable (key, sec) order in the key range."""
    from horsepower_gb300 import data as D, plans as P, serve as S
    gpu = libs[0]
    rng = np.random.default_rng(nreq)
    line = S.line_table(gpu, 50_021, seed=nreq)
    from horsepower_gb300 import batch as B
    dim, fact = B.device_tables(gpu, *D.join_tables(nfact=3000, ndim=700, seed=3))
    n = 200_003
    key = np.minimum(rng.zipf(1.2, n), 1 << 40).astype(np.int64)
    sec = rng.integers(0, 1000, n).astype(np.int32)
    order = dict(key=B.to_device(gpu, key, H_L), sec=B.to_device(gpu, sec, H_I))
    srv = S.Server(gpu, line, dim, fact, order, budget=1 << 30)
    reqs = []
    for _ in range(nreq):
        lo = int(D.DAYS0 + rng.integers(0, D.NDAYS))
        reqs.append(S.Request(S.FILTER_AGG, lo, lo + int(rng.integers(0, 900)), 0, 0, 0.0))
        a = int(rng.choice([1, 2, 50, 10_000, 1 << 30]))
        reqs.append(S.Request(S.TOPK_ORDER, 0, 0, a, a + int(rng.choice([0, 1, 100, 1 << 35])), 0.0))
    got, _, _ = srv.run(reqs)
    for r, v in zip(reqs, got):
        if r.kind == S.FILTER_AGG:
            ch = P.Chain(gpu, P.Q6_CHAIN.format(lo=r.lo, hi=r.hi)) if nreq < 10 else None
            if ch:
                f = gpu.to_py(ch.run([line["shipdate"], line["qty"], line["disc"], line["price"]]))[0]
                assert v == f, (r.lo, r.hi)
        else:
            rows = np.flatnonzero((key >= r.klo) & (key < r.khi))
            want = rows[np.lexsort((sec[rows], key[rows]))][: S.TOPK]
            assert np.array_equal(v, want), (r.klo, r.khi)
    srv.close()
    gpu.free_inputs()


@pytest.mark.parametrize("typ", [H_B, H_J, H_H, H_I, H_L, H_F, H_E])
@pytest.mark.parametrize("n", [2, 15, 31, 511, 512, 513, 4096 + 7, 70_001])
def test_elementwise_chunks(libs, typ, n):
    """Compare, arithmetic, logic and not around the 512-element chunks, from
    16-byte-aligned columns and from views that start one element later, for
    vector and scalar operands on either side: equal to the oracle."""
    from horsepower_gb300 import batch as B
    gpu, ora = libs
    rng = np.random.default_rng(n + typ)
    dt = DTYPE[typ]
    cols = []
    for _ in range(2):
        if typ == H_B:
            cols.append(rng.random(n + 1) < 0.5)
        elif typ in (H_F, H_E):
            c = np.round(rng.standard_normal(n + 1), 1).astype(dt)
            c[rng.random(n + 1) < 0.05] = np.nan
            cols.append(c)
        else:
            cols.append(rng.integers(-5, 6, n + 1).astype(dt))
    names = ["pfnLt", "pfnLeq", "pfnGt", "pfnGeq", "pfnEq", "pfnNeq", "pfnPlus", "pfnMinus", "pfnMul"]
    names += ["pfnAnd", "pfnOr", "pfnXor", "pfnNand", "pfnNor"] if typ == H_B else ["pfnDiv"]
    for skip in (0, 1):
        a, b = cols[0][skip:], cols[1][skip:]
        if typ != H_B:
            b = np.where(b == 0, dt(3), b)      # divisors
        s = b[0] if b[0] == b[0] else dt(0.1)

        def view(c, skip=skip):
            d = B.to_device(gpu, np.concatenate([c[:1]] * skip + [c]), typ)
            d.g, d.len = d.g + skip * c.itemsize, c.size
            return d

        da, db = view(a), view(b)
        for f in names:
            for x, y, hx, hy in ((da, db, a, b), (da, s, a, s), (s, db, s, b)):
                dev = [gpu.scalar(v, typ) if isinstance(v, np.generic) else v for v in (x, y)]
                host = [ora.scalar(v, typ) if isinstance(v, np.generic) else ora.vec(v, typ) for v in (hx, hy)]
                got, want = gpu.to_py(gpu.call(f, *dev)), ora.to_py(ora.call(f, *host))
                assert got.dtype == want.dtype and np.array_equal(got, want, equal_nan=got.dtype.kind == "f"), (f, skip)
        if typ == H_B:
            assert np.array_equal(gpu.to_py(gpu.call("pfnNot", da)), ~a)
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("n", [1, 255, 1023, 1025, 4096, 4097, 50_001])
@pytest.mark.parametrize("text,typs", [
    ("(sum (mul x2 x1) (and (lt x0 3:i32) (gt x1 0.25:f64)))", (H_I, H_E, H_E)),   # a value column the mask also reads
    ("(max x1 (lt x0 x2))", (H_H, H_F, H_J)),
    ("(min x0 (neq x0 2:i64))", (H_L,)),
    ("(count (or x0 (lt x1 0:i32)))", (H_B, H_I)),
])
def test_chain_rounds(libs, n, text, typs):
    """A fused reduction's rounds of four rows, last tile ragged, one and
    several tiles: the f64 sum bit-identical to the fixed tile tree over the
    rows with unselected ones as -0.0, the others to numpy."""
    from horsepower_gb300 import plans as P
    gpu, ora = libs
    rng = np.random.default_rng(n)
    x = [rng.random(n) < 0.3 if t == H_B else (rng.standard_normal(n).astype(DTYPE[t]) if t in (H_F, H_E)
         else rng.integers(-9, 10, n).astype(DTYPE[t])) for t in typs]
    got = gpu.to_py(P.Chain(gpu, text).run([gpu.vec(c, t) for c, t in zip(x, typs)]))[0]
    if text.startswith("(sum"):
        m = (x[0] < 3) & (x[1] - 0.25 >= 1e-13)
        v = np.where(m, x[2] * x[1], -0.0)
        want = ora.lib.hgoTreeSumF64(np.ascontiguousarray(v).ctypes.data, n)
        assert got == want, (got, want)
    elif text.startswith("(max"):
        m = x[0] < x[2]
        if m.any():
            assert got == x[1][m].max()
    elif text.startswith("(min"):
        if (x[0] != 2).any():
            assert got == x[0][x[0] != 2].min()
    else:
        assert got == (x[0] | (x[1] < 0)).sum()
    gpu.free_inputs()


@pytest.mark.parametrize("copies", [1, 7, 33])
def test_small_groups(libs, copies):
    """Groups of 1 to 33 rows, any number of each size: sums equal the fixed
    tile tree of their rows bit for bit, min and max follow the xor butterfly's
    operand order (which decides where NaN goes)."""
    gpu, ora = libs
    rng = np.random.default_rng(copies)
    sizes = np.repeat(np.arange(1, 34), copies)
    key = np.repeat(np.arange(sizes.size, dtype=np.int32), sizes)
    rng.shuffle(key)
    pay = rng.standard_normal(key.size) * 10.0 ** rng.integers(-8, 8, key.size)
    pay[rng.random(key.size) < 0.05] = -0.0
    nanp = np.where(rng.random(key.size) < 0.2, np.nan, pay)
    g = gpu.call("pfnGroup", gpu.vec(key, H_I))
    vals, keys = gpu.call("pfnValues", g), gpu.to_py(gpu.call("pfnKeys", g))
    sums = gpu.to_py(gpu.call("hgpuGroupSum", gpu.vec(pay, H_E), vals))
    isum = gpu.to_py(gpu.call("hgpuGroupSum", gpu.vec(key, H_I), vals))
    lo = gpu.to_py(gpu.call("hgpuGroupMin", gpu.vec(nanp, H_E), vals))
    hi = gpu.to_py(gpu.call("hgpuGroupMax", gpu.vec(nanp, H_E), vals))

    def butterfly(x, op, ident):
        p = 1 << max(0, (len(x) - 1).bit_length())
        x = [op(ident, v) for v in x] + [ident] * (p - len(x))
        while p > 1:
            p //= 2
            x = [op(x[j], x[j + p]) for j in range(p)]
        return x[0]

    top = np.inf
    for gi, first in enumerate(keys):
        rows = np.flatnonzero(key == key[first])
        x = np.ascontiguousarray(pay[rows])
        want = ora.lib.hgoTreeSumF64(x.ctypes.data, x.size)
        assert sums[gi].tobytes() == np.float64(want).tobytes(), (len(rows), sums[gi], want)
        assert isum[gi] == len(rows) * int(key[first])
        if len(rows) <= 32:
            for got, op, ident in ((lo[gi], lambda a, b: a if a < b else b, top),
                                   (hi[gi], lambda a, b: a if a > b else b, -top)):
                want = butterfly(list(nanp[rows]), op, ident)
                assert got == want or (got != got and want != want), (len(rows), got, want)
    gpu.free_inputs()


@pytest.mark.parametrize("nplans,nfact", [(32, 30_001), (33, 5_000), (40, 120_013)])
def test_shared_many_windows(libs, nplans, nfact):
    """As many windows as one pass over the fact table takes, and more (random
    ends, all distinct or shared, empty and full windows among them): each
    plan's rows equal the same plan alone, bit for bit."""
    from horsepower_gb300 import batch as B, data as D, plans as P
    gpu = libs[0]
    dim, fact = D.join_tables(nfact=nfact, ndim=max(2, nfact // 4), seed=nplans)
    rng = np.random.default_rng(nplans)
    ddim, dfact = B.device_tables(gpu, dim, fact)
    ends = np.sort(rng.integers(D.DAYS0 - 5, D.DAYS0 + 2531, (nplans, 2)), axis=1)
    ends[0], ends[1], ends[2] = (D.DAYS0, D.DAYS0 + 2526), (9000, 9000), ends[3]
    got = B.run_batch(gpu, [B.make_plan(ddim, dfact, int(lo), int(hi)) for lo, hi in ends])
    for (lo, hi), r in zip(ends, got):
        sel = dim["pk"][(dim["date"] >= lo) & (dim["date"] < hi)]
        if not np.isin(fact["fk"], sel).any():
            assert len(r[0]) == 0
            continue
        for a, b in zip(r, P.join_group(gpu, ddim, dfact, int(lo), int(hi))):
            assert np.array_equal(a, gpu.to_py(b)), (lo, hi)
    gpu.free_inputs()


@pytest.mark.parametrize("n,kind", [
    (4097, "random"), (65_536, "few"), (311_296, "random"), (311_297, "few"), (622_592, "random"), (622_593, "random"),
    (5_000, "sorted"), (9_000, "organ"),                         # deeper than one launch runs
])
def test_quicksort_depths(libs, n, kind):
    """Quicksort orders whose partitions above one CTA's size run in one launch
    of resident blocks (two or four elements a thread, or past them with four
    launches a depth), and recursions deeper than a launch: the reference's
    order of equal keys, both directions."""
    gpu, ora = libs
    rng = np.random.default_rng(n)
    x = {"random": lambda: rng.standard_normal(n), "few": lambda: rng.integers(0, 40, n) / 8.0,
         "sorted": lambda: np.arange(n) / 3.0, "organ": lambda: np.minimum(np.arange(n), n - np.arange(n)) * 1.0}[kind]()
    for up in (True, False):
        d = np.array([up])
        a = gpu.to_py(gpu.call("pfnOrderBy", gpu.vec(x, H_E), gpu.vec(d, H_B)))
        b = ora.to_py(ora.call("pfnOrderBy", ora.vec(x, H_E), ora.vec(d, H_B)))
        assert np.array_equal(a, b), up
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("n", [4096, 5000, 300_001])
@pytest.mark.parametrize("lo,hi,mul", [(-70_000, -1, 1), (-70_000, 70_000, 1), (0, 70_000, 1 << 12), (1 << 30, (1 << 30) + 9, 1),
                                       (-1, 1, 1 << 31), (5, 6, 1)])
def test_group_key_stats(libs, n, lo, hi, mul):
    """@group of i32 and i64 keys whose varying bits come with their range:
    negative, mixed signs, constant low bits, constant bits inside, one value.
    Keys and row lists are those of the stable sort of the reference's order."""
    gpu, ora = libs
    rng = np.random.default_rng(n)
    for typ in (H_I, H_L):
        key = rng.integers(lo, hi, n) * mul
        if typ == H_I:
            key = key.astype(np.int32).astype(np.int64)
        key = key.astype(DTYPE[typ])
        a, b = gpu.call("pfnGroup", gpu.vec(key, typ)), ora.call("pfnGroup", ora.vec(key, typ))
        assert np.array_equal(gpu.to_py(gpu.call("pfnKeys", a)), ora.to_py(ora.call("pfnKeys", b))), typ
        for x, y in zip(gpu.to_py(gpu.call("pfnValues", a)), ora.to_py(ora.call("pfnValues", b))):
            assert np.array_equal(x, y)
        gpu.free_inputs()
        ora.free_inputs()


@pytest.mark.parametrize("tiles", [1, 2, 255, 257, 2047, 2048, 2049])
@pytest.mark.parametrize("cut", [0, 1, 4095])
def test_compact_offsets(libs, tiles, cut):
    """@where and @compress with as many tiles as find their offsets
    themselves, and more: against numpy, rows selected up to the last."""
    gpu = libs[0]
    n = tiles * 4096 - cut
    rng = np.random.default_rng(tiles + cut)
    m = rng.random(n) < 0.01
    m[-1] = True
    v = np.arange(n, dtype=np.int16)
    dm = gpu.vec(m, H_B)
    assert np.array_equal(gpu.to_py(gpu.call("pfnWhere", dm)), np.flatnonzero(m))
    assert np.array_equal(gpu.to_py(gpu.call("pfnCompress", dm, gpu.vec(v, H_H))), v[m])
    gpu.free_inputs()


def test_topk_sizes(libs):
    """Top-k requests with 1 to more than 4096 candidates (one CTA sorts up to
    4096; ties on the key, the second column and the row), negative keys and
    second columns: the first rows of the stable order."""
    from horsepower_gb300 import batch as B, data as D, serve as S
    gpu = libs[0]
    rng = np.random.default_rng(5)
    counts = [1, 2, 3, 31, 33, 999, 1000, 1001, 2047, 2048, 2049, 4095, 4096, 4097, 9000]
    key = np.repeat(np.arange(len(counts), dtype=np.int64) * 3 - 20, counts)
    sec = rng.choice(np.array([-2 ** 31, -7, 0, 5, 2 ** 31 - 1]), key.size).astype(np.int32)
    p = rng.permutation(key.size)
    key, sec = key[p], sec[p]
    line = S.line_table(gpu, 5000, seed=1)
    dim, fact = B.device_tables(gpu, *D.join_tables(nfact=300, ndim=70, seed=3))
    srv = S.Server(gpu, line, dim, fact, dict(key=B.to_device(gpu, key, H_L), sec=B.to_device(gpu, sec, H_I)), budget=1 << 30)
    reqs = [S.Request(S.TOPK_ORDER, 0, 0, int(k), int(k) + w, 0.0) for k in np.unique(key) for w in (1, 4, 100)]
    got, _, _ = srv.run(reqs)
    for r, v in zip(reqs, got):
        rows = np.flatnonzero((key >= r.klo) & (key < r.khi))
        want = rows[np.lexsort((rows, sec[rows], key[rows]))][: S.TOPK]
        assert np.array_equal(v, want), (r.klo, r.khi)
    srv.close()
    gpu.free_inputs()


@pytest.mark.parametrize("typ", [H_H, H_I, H_L, H_F, H_E])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 70_001])
@pytest.mark.parametrize("wide", [False, True])
def test_member_rounds(libs, typ, n, wide):
    """@member in rounds of eight keys a lane, sets of a narrow range (the
    presence bit answers) and of a wide one (hashed), keys outside the range
    and NaN: equal to the oracle."""
    gpu, ora = libs
    rng = np.random.default_rng(n + typ)
    span = {H_H: 30_000, H_I: 2 ** 31 - 1, H_L: 2 ** 62, H_F: 1e6, H_E: 1e9}[typ] if wide else 3000
    make = lambda m, s: (rng.integers(-s, s, m) if typ in (H_H, H_I, H_L) else np.round(rng.uniform(-s, s, m))).astype(DTYPE[typ])  # noqa: E731
    x = make(1000, span)
    y = np.where(rng.random(n) < 0.5, rng.choice(x, n), make(n, min(4 * span, 32_000) if typ == H_H else span))
    if typ in (H_F, H_E):
        x[3] = np.nan
        y[rng.random(n) < 0.1] = np.nan
    y = y.astype(DTYPE[typ])
    a = gpu.to_py(gpu.call("pfnMember", gpu.vec(x, typ), gpu.vec(y, typ)))
    b = ora.to_py(ora.call("pfnMember", ora.vec(x, typ), ora.vec(y, typ)))
    assert np.array_equal(a, b)
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("ndim,span", [(2, 2), (7, 8), (255, 2040), (1000, 63_999)])
@pytest.mark.parametrize("repeat", [False, True])
def test_shared_probe_keys(libs, ndim, span, repeat):
    """The shared date table filled by plain stores: key ranges with empty
    places and odd lengths, negative keys, and a repeated key, which sends the
    plans to their builtins.  Fact keys outside the dimension match nothing."""
    from horsepower_gb300 import batch as B, data as D, plans as P
    gpu = libs[0]
    dim, fact = D.join_tables(nfact=5000, ndim=ndim, seed=ndim)
    rng = np.random.default_rng(span)
    dim["pk"] = (rng.choice(span, ndim, replace=False) - span // 2).astype(np.int32)
    if repeat:
        dim["pk"][-1] = dim["pk"][0]
    fact["fk"] = np.where(rng.random(5000) < 0.9, rng.choice(dim["pk"], 5000), span).astype(np.int32)
    ddim, dfact = B.device_tables(gpu, dim, fact)
    wins = [(D.DAYS0, D.DAYS0 + 2526), (D.DAYS0 + 100, D.DAYS0 + 1500), (D.DAYS0, D.DAYS0 + 2526)]
    got = B.run_batch(gpu, [B.make_plan(ddim, dfact, lo, hi) for lo, hi in wins])
    for (lo, hi), r in zip(wins, got):
        if not np.isin(fact["fk"], dim["pk"][(dim["date"] >= lo) & (dim["date"] < hi)]).any():
            assert len(r[0]) == 0
            continue
        for a, b in zip(r, P.join_group(gpu, ddim, dfact, lo, hi)):
            assert np.array_equal(a, gpu.to_py(b)), (lo, hi)
    gpu.free_inputs()


@pytest.mark.parametrize("codes", [1, 2, 31, 255, 256, 257, 300])
@pytest.mark.parametrize("n", [4096, 8191, 150_001])
def test_group_few_codes(libs, codes, n):
    """@group of i32 keys with few values in a narrow range (the counting path,
    its rank table made on the device, one or several rounds of the scan) and
    with one too many: keys and row lists of the stable order."""
    gpu = libs[0]
    rng = np.random.default_rng(codes)
    vals = np.sort(rng.choice(60_000, codes, replace=False)).astype(np.int32)
    key = rng.choice(vals, n)
    key[:codes] = vals
    g = gpu.call("pfnGroup", gpu.vec(key, H_I))
    order = np.argsort(key, kind="stable")
    starts = np.flatnonzero(np.r_[True, np.diff(key[order]) != 0])
    assert np.array_equal(gpu.to_py(gpu.call("pfnKeys", g)), order[starts])
    lists = gpu.to_py(gpu.call("pfnValues", g))
    assert len(lists) == codes
    for a, b in zip(lists, np.split(order, starts[1:])):
        assert np.array_equal(a, b)
    gpu.free_inputs()
