"""Rules that choose between kernels: which kernels a call launches on either
side of a rule's line, and that its result is the same on both.

Bar: bit-exact.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from horsepower_gb300.abi import Builtins, DTYPE, H_B, H_E, H_F, H_H, H_I, H_J, H_L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import horsepower_gb300
    L = horsepower_gb300.load()
    L.lib.hgpuProfileRead.argtypes = [C.c_int32, C.POINTER(C.c_char_p), C.POINTER(C.c_double), C.POINTER(C.c_longlong)]
    return L


@pytest.fixture(scope="module")
def ora():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run(["make", "-s", "-C", os.path.join(root, "oracle"), "port"], check=True)
    return Builtins(os.path.join(root, "oracle", "_build", "liboracle.so"), "oracle")


def launches(L, fn):
    """fn()'s result and its launches by kernel name."""
    L.lib.hgpuProfileReset()
    L.lib.hgpuProfile(1)
    try:
        out = fn()
    finally:
        L.lib.hgpuProfile(0)
    names, ms, n = (C.c_char_p * 256)(), (C.c_double * 256)(), (C.c_longlong * 256)()
    k = L.lib.hgpuProfileRead(256, names, ms, n)
    got = {names[i].decode(): n[i] for i in range(k)}
    L.lib.hgpuProfileReset()
    return out, got


@pytest.mark.parametrize("n", [3, 255, 257, 2048 + 5, 70_001])
@pytest.mark.parametrize("typ,span,kernel", [(H_I, 4000, "member"), (H_H, 30_000, "member"), (H_L, 60_000, "member"),
                                             (H_I, 2 ** 31 - 1, "member_hash"), (H_L, 2 ** 62, "member_hash"),
                                             (H_F, 0, "member_hash"), (H_E, 0, "member_hash")])
def test_member_routes(gpu, typ, span, kernel, n):
    """@member looks eight keys up at a time in a direct table and one at a
    time in a hashed one, where eight take the registers that hide the walk."""
    rng = np.random.default_rng(n + typ)
    if span:
        x, other = (rng.integers(-span // 2, span // 2, m).astype(DTYPE[typ]) for m in (1000, n))
        x[:2] = [-(span // 2), span // 2 - 1]
    else:
        x, other = (rng.standard_normal(m).astype(DTYPE[typ]) for m in (1000, n))
        other[::7] = np.nan
    y = np.where(rng.random(n) < 0.5, rng.choice(x, n), other)
    z, got = launches(gpu, lambda: gpu.call("pfnMember", gpu.vec(y, typ), gpu.vec(x, typ)))
    assert np.array_equal(gpu.to_py(z), np.isin(y, x))
    assert {k for k in got if k.startswith("member")} == {kernel}, got
    gpu.free_inputs()


def order(L, x, asc=True):
    return L.to_py(L.call("pfnOrderBy", L.vec(x, H_E), L.vec(np.array([asc]), H_B)))


@pytest.mark.parametrize("n", [2048 * 4096, 2048 * 4096 + 1, 2048 * 4103 + 77])
def test_quicksort_tile_sums(gpu, ora, n):
    """Above 4096 tiles the tile sums of a quicksort depth are scanned by a
    kernel of their own instead of added up by every block; keys with ties,
    so that the permutation is the sequential quicksort's and no other."""
    x = np.random.default_rng(n).integers(0, n // 2, n) * 0.5
    got, k = launches(gpu, lambda: order(gpu, x))
    assert ("qs_scan_sums" in k) == (n > 2048 * 4096), k
    assert np.array_equal(got, order(ora, x))
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("values", [1, 3, 5])
def test_quicksort_few_values(gpu, ora, values):
    """Keys of few values are sorted after a few depths: no more than the first
    round of depths is issued for them."""
    n = 700_001
    x = np.random.default_rng(values).integers(0, values, n) * 0.5
    got, k = launches(gpu, lambda: order(gpu, x))
    assert 0 < k["qs_count"] <= 8, k
    assert np.array_equal(got, order(ora, x))
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("copies,kernels", [(7, {"qs_blocks"}), (200, {"qs_blocks", "qs_blocks_128", "qs_blocks_512"})])
def test_quicksort_classes(gpu, ora, copies, kernels):
    """Segments of a list order on either side of what a CTA of 32, 128 and
    1024 threads holds: many of a size have a launch of their own, few go with
    the larger ones.  Keys with ties, some segments of one value or ordered."""
    sizes = np.tile([32, 33, 64, 127, 128, 129, 200, 511, 512, 513, 1024, 4095, 4096], copies)
    rng = np.random.default_rng(copies)
    rng.shuffle(sizes)
    seg = np.repeat(np.arange(sizes.size, dtype=np.int32), sizes)
    key = rng.integers(0, 60, seg.size) * 0.5
    key[np.isin(seg, np.arange(0, sizes.size, 11))] = 2.0
    rising = np.isin(seg, np.arange(3, sizes.size, 13))
    key[rising] = np.arange(rising.sum())
    mix = rng.permutation(seg.size)
    seg, key = seg[mix], key[mix]

    def run(L, up=(True, True)):
        return L.to_py(L.call("pfnOrderBy", L.list([L.vec(seg, H_I), L.vec(key, H_E)]), L.vec(np.array(up), H_B)))

    got, k = launches(gpu, lambda: run(gpu))
    assert {x for x in k if x.startswith("qs_blocks")} == kernels, k
    assert np.array_equal(got, run(ora))
    assert np.array_equal(run(gpu, (True, False)), run(ora, (True, False)))
    gpu.free_inputs()
    ora.free_inputs()


@pytest.mark.parametrize("n", [304 * 4096, 304 * 4096 + 1, 1_600_003, 2 * 304 * 4096 + 511])
@pytest.mark.parametrize("form", ["vv", "vs", "sv"])
def test_arith_spread(gpu, n, form):
    """f64 division over more blocks than the SMs hold at once: the chunks are
    spread over them, the last one ragged; a zero divisor in it is found."""
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    b[b == 0] = 1.0
    x = gpu.vec(a, H_E) if form[0] == "v" else gpu.scalar(a[0], H_E)
    y = gpu.vec(b, H_E) if form[1] == "v" else gpu.scalar(b[0], H_E)
    ha, hb = (a if form[0] == "v" else a[0]), (b if form[1] == "v" else b[0])
    for f, want in (("pfnPlus", ha + hb), ("pfnMinus", ha - hb), ("pfnMul", ha * hb), ("pfnDiv", ha / hb)):
        z, k = launches(gpu, lambda: gpu.call(f, x, y))
        assert np.array_equal(gpu.to_py(z), want), f
        assert ("arith_spread" in k) == (f == "pfnDiv" and n > 304 * 4096), k
    if form[1] == "v":
        b[n - 1] = 0.0
        assert gpu.rc("pfnDiv", x, gpu.vec(b, H_E)) == 4  # E_DIV_ZERO
    gpu.free_inputs()


@pytest.mark.parametrize("n", [1, 4097, 70_001])
def test_chain_many_columns(gpu, n):
    """A chain of more than 1024 columns takes its pointers from device memory
    instead of the kernel's parameters: each kind of sink against numpy."""
    from horsepower_gb300 import plans as P
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal(n), rng.integers(-9, 10, n).astype(np.int32)
    cols = [gpu.vec(a, H_E)] + [gpu.vec(b, H_I)] * 1028 + [gpu.vec(2 * a, H_E)]
    assert len(cols) == 1030

    def run(text, many=0):
        ch = P.Chain(gpu, text)
        return [gpu.to_py(z) for z in (ch.run_many(cols, many) if many else [ch.run(cols)])]

    keep = b > 2
    got = run("(map (plus x0 x1029) (plus x1028 1:i32))", 2)
    assert np.array_equal(got[0], a + 2 * a) and np.array_equal(got[1], b + 1)
    got = run("(compress (gt x1000 2:i32) (mul x1029 x0) x7)", 2)
    assert np.array_equal(got[0], (2 * a * a)[keep]) and np.array_equal(got[1], b[keep])
    assert run("(count (gt x1000 2:i32))")[0] == keep.sum()
    assert run("(sum (mul x1 x1028) (gt x1000 2:i32))")[0] == (b.astype(np.int64) ** 2)[keep].sum()
    if keep.any():
        assert run("(max x1029 (gt x1000 2:i32))")[0] == (2 * a)[keep].max()
    gpu.free_inputs()


@pytest.mark.parametrize("n", [2, 3071, 3072, 3073, 9216 + 5, 200_003])
@pytest.mark.parametrize("shape", ["both signs", "one positive", "a constant bit"])
def test_radix_signed_keys(gpu, n, shape):
    """@order and @group of i64 keys in which 63 or 64 bits vary, the sign among
    them: key and row id never fit one record, so these take the passes over two
    arrays.  With a value of 2^32 or more the order is that of the unsigned
    words, negatives behind the others; either direction, every digit, whole
    and ragged tiles."""
    rng = np.random.default_rng(n + len(shape))
    key = rng.integers(-2 ** 63, 2 ** 63, n, dtype=np.int64)
    key[rng.random(n) < 0.3] = key[0]
    if shape == "one positive":
        key = (key.view(np.uint64) | np.uint64(2 ** 63)).view(np.int64)
        key[n // 2] = 2 ** 63 - 1
    elif shape == "a constant bit":
        key &= ~np.int64(32)
        key[:2] = [-2 ** 63, 2 ** 63 - 1 - 32]
    else:
        key[:2] = [-2 ** 63, 2 ** 63 - 1]
    rng.shuffle(key)
    want = np.argsort(key.view(np.uint64), kind="stable")
    k = gpu.vec(key, H_L)
    up, names = launches(gpu, lambda: gpu.to_py(gpu.call("pfnOrderBy", k, gpu.vec(np.array([1], bool), H_B))))
    assert np.array_equal(up, want)
    assert n == 2 or names["radix_scatter"] == 8, names  # (of two keys fewer bits may vary)
    down = gpu.to_py(gpu.call("pfnOrderBy", k, gpu.vec(np.array([0], bool), H_B)))
    assert np.array_equal(down, want[::-1])
    if n < 20_000:
        g = gpu.to_py(gpu.call("pfnGroup", k))
        heads = np.flatnonzero(np.r_[True, key[want][1:] != key[want][:-1]])
        assert np.array_equal(g[1], want[heads])
        assert np.array_equal(np.concatenate(g[2]), want)
    gpu.free_inputs()


@pytest.mark.parametrize("n", [2, 511, 512, 513, 4096 + 7, 70_001])
@pytest.mark.parametrize("typ", [H_B, H_J, H_H, H_I, H_L, H_F, H_E])
def test_one_unaligned_operand(gpu, typ, n):
    """An operand that does not begin on 16 bytes is read element by element
    beside one that is read 16 bytes at a time: the results of every
    combination are those of two aligned columns."""
    from horsepower_gb300 import batch as B
    rng = np.random.default_rng(n + typ)
    a, b = (rng.integers(0, 2 if typ == H_B else 100, n).astype(DTYPE[typ]) for _ in range(2))

    def column(c, skip):
        d = B.to_device(gpu, np.concatenate([c[:1]] * skip + [c]), typ)
        d.g, d.len = d.g + skip * c.itemsize, n
        return d

    names = ["pfnLt", "pfnEq", "pfnPlus", "pfnMul"] + (["pfnAnd", "pfnXor"] if typ == H_B else [])
    s = gpu.scalar(1, typ)
    for f in names:
        def run(da, db):
            return [gpu.to_py(gpu.call(f, x, y)).tobytes() for x, y in ((da, db), (da, s), (s, db))]
        want = run(column(a, 0), column(b, 0))
        for sa, sb in ((1, 0), (0, 1), (1, 3), (5, 5)):
            assert run(column(a, sa), column(b, sb)) == want, (f, sa, sb)
    gpu.free_inputs()


@pytest.mark.parametrize("length,every,short,walks", [
    (513, 0, 0, True),          # every round's eight segments are long
    (640, 97, 40, True),        # most rounds'
    (1100, 3, 512, True),       # none: a third of the segments is not
    (513, 2, 33, False),        # the class averages fewer than 512 rows
])
def test_long_mid_segments_walk(gpu, ora, length, every, short, walks):
    """More mid-size segments than one round of the grid takes, long on
    average: rounds of eight segments above 512 rows go to a kernel in which
    each warp walks one.  i64 sums and maxima equal numpy's, f64 sums the fixed
    tile tree of their rows, in rounds of either kind."""
    ora.lib.hgoTreeSumF64.restype = C.c_double
    ora.lib.hgoTreeSumF64.argtypes = [C.c_void_p, C.c_longlong]
    groups = 32 * 8 * 152 + 1003
    sizes = np.full(groups, length)
    if every:
        sizes[::every] = short
    rng = np.random.default_rng(length)
    key = np.repeat(np.arange(groups, dtype=np.int32), sizes)
    key = np.roll(key, 12_345)          # groups are found by value, not by place
    n = key.size
    pay = rng.standard_normal(n) * 10.0 ** rng.integers(-6, 6, n)
    ipay = rng.integers(-2 ** 62, 2 ** 62, n)
    vals = gpu.call("pfnValues", gpu.call("pfnGroup", gpu.vec(key, H_I)))
    dpay, dipay = gpu.vec(pay, H_E), gpu.vec(ipay, H_L)
    sums, ran = launches(gpu, lambda: gpu.to_py(gpu.call("hgpuGroupSum", dpay, vals)))
    assert ("seg_walk" in ran) == walks, ran
    isums = gpu.to_py(gpu.call("hgpuGroupSum", dipay, vals))
    imax = gpu.to_py(gpu.call("hgpuGroupMax", dipay, vals))
    order = np.argsort(key, kind="stable")
    starts = np.r_[0, np.cumsum(sizes)[:-1]]
    assert np.array_equal(isums, np.add.reduceat(ipay[order], starts))
    assert np.array_equal(imax, np.maximum.reduceat(ipay[order], starts))
    for g in np.r_[:20, rng.integers(0, groups, 400), groups - 20:groups]:
        x = np.ascontiguousarray(pay[order[starts[g]:starts[g] + sizes[g]]])
        want = ora.lib.hgoTreeSumF64(x.ctypes.data, x.size)
        assert sums[g].tobytes() == np.float64(want).tobytes(), (g, sizes[g])
    gpu.free_inputs()
