"""The calls this library is timed on, at the sizes a query engine makes them.

A user of libhgpu is the HorseIR interpreter or the C code its compiler
generates: a query is a sequence of builtin calls over columns that are
already in HBM, and its results are small or large vectors.  The kinds of
case are the benchmark's configurations (`bench.py`), each over the range of
table sizes from a few tens of thousands of rows to the full tables, and the
two orderings and the semi-join that TPC-H-shaped queries
(`horsepower_gb300/plans.py`) end or begin with:

  filter_agg    the q6 filter and sum, one builtin call per statement
  filter_fused  the same as one compiled chain (`hgpuChainRun`)
  join_group    dimension filter, join, gathers, @group, four aggregates: the
                query compiled to C
  group_agg     @group of one key column, per-group sum and count
  order_pair    stable ascending @order of (key, secondary)
  order_top     ORDER BY revenue desc, date: @order of an (f64, i32) pair and
                the gathers by it
  semi_join     @member mask, @compress by it, avg / min / max of the selection
  batch         many join + group-by plans over tables of their own in one call
  serve         one admission step of the request loop over resident tables

Every pass runs through the public entry points with a heap rewind before
it, as a query engine does between queries.  Inputs are torch tensors made
on the device from the seed; a window of dates is part of the query, not of
the data, so all seeds of a case share it.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import horsepower_gb300
from horsepower_gb300 import batch as B
from horsepower_gb300 import data as D
from horsepower_gb300 import plans as P
from horsepower_gb300 import serve as S
from horsepower_gb300.abi import H_B, H_C, H_E, H_I, H_L, V0

LINE_ROWS = 6_001_215      # the filter table of the first configuration
FACT_ROWS = 59_986_052     # the fact table of the second
DIM_ROWS = 15_000_000
GROUP_ROWS = 150_000_000   # the third configuration's table
GROUP_RANKS = 10_000_000


def listed():
    return [
        # a selective query over a small table: 13 calls, all of it launches and waits
        dict(name="filter_agg_60K", kind="filter_agg", rows=60_175),
        # the first configuration's table, one builtin call per statement
        dict(name="filter_agg_6M", kind="filter_agg", rows=LINE_ROWS),
        # the same filter as the optimizer's fused loop, over a large table
        dict(name="filter_fused_60M", kind="filter_fused", rows=FACT_ROWS),
        # the join + group-by query over a table a hundredth of the full one
        dict(name="join_group_600K", kind="join_group", rows=599_861, dim=150_000),
        # the second configuration in full: the benchmark's headline query
        dict(name="join_group_60M", kind="join_group", rows=FACT_ROWS, dim=DIM_ROWS),
        # GROUP BY on an ordinary intermediate result, i32 keys
        dict(name="group_agg_1_5M", kind="group_agg", rows=1_500_003, ranks=100_000, key="i32"),
        # the third configuration's grouping in full: Zipf i64 keys
        dict(name="group_agg_150M", kind="group_agg", rows=GROUP_ROWS, ranks=GROUP_RANKS, key="i64"),
        # the third configuration's order in full: (i64 key, i32 secondary)
        dict(name="order_pair_150M", kind="order_pair", rows=GROUP_ROWS, ranks=GROUP_RANKS, key="i64"),
        # ORDER BY revenue desc, date over the groups a query ends with
        dict(name="order_top_114K", kind="order_top", rows=114_003),
        # EXISTS / IN over the fact table's foreign key, then statistics of the selection
        dict(name="semi_join_60M", kind="semi_join", rows=FACT_ROWS, dim=DIM_ROWS),
        # 64 independent small and middling plans in one call
        dict(name="batch_64", kind="batch", plans=64, lo=10_000, hi=4_000_000),
        # one step of the served form over the full tables: 64 waiting requests
        dict(name="serve_64", kind="serve", requests=64, line=LINE_ROWS, rows=FACT_ROWS, dim=DIM_ROWS,
             order=GROUP_ROWS),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["filter_agg", "filter_fused", "join_group", "group_agg", "group_agg", "order_pair",
                       "order_pair", "order_top", "semi_join", "batch", "serve"])
    if kind == "filter_agg":
        return dict(kind=kind, rows=log(60_000, LINE_ROWS))
    if kind == "filter_fused":
        return dict(kind=kind, rows=log(60_000, FACT_ROWS))
    if kind in ("join_group", "semi_join"):
        rows = log(100_000, FACT_ROWS)
        return dict(kind=kind, rows=rows, dim=max(1000, rows // rng.choice([3, 4, 5, 8])))
    if kind in ("group_agg", "order_pair"):
        rows = log(100_000, GROUP_ROWS)
        return dict(kind=kind, rows=rows, ranks=log(1000, max(2000, rows // 15)), key=rng.choice(["i32", "i64"]))
    if kind == "order_top":
        return dict(kind=kind, rows=log(3_000, 114_000))
    if kind == "batch":
        return dict(kind=kind, plans=rng.randrange(8, 65), lo=10_000, hi=log(100_000, 4_000_000))
    rows = log(600_000, FACT_ROWS)
    return dict(kind=kind, requests=rng.randrange(8, 65), line=log(60_000, LINE_ROWS), rows=rows, dim=rows // 4,
                order=log(1_000_000, GROUP_ROWS))


# ------------------------------------------------------------------- tables
DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _ints(g, lo, hi, n, dtype):
    return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=dtype)


def _uniform(g, lo, hi, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _measures(g, qty):
    """price and disc as `horsepower_gb300.data` draws them."""
    price = torch.round(qty.double() * _uniform(g, 900.0, 105000.0, qty.numel())) / 100.0
    disc = _ints(g, 0, 11, qty.numel(), torch.int32).double() / 100.0
    return price, disc


def _line(g, n):
    qty = _ints(g, 1, 51, n, torch.int32)
    price, disc = _measures(g, qty)
    return dict(shipdate=_ints(g, D.DAYS0, D.DAYS0 + D.NDAYS, n, torch.int32), qty=qty, disc=disc, price=price)


def _join(g, n, ndim):
    dim = dict(pk=torch.randperm(ndim, generator=g, device=DEV, dtype=torch.int32),
               date=_ints(g, D.DAYS0, D.DAYS0 + D.NDAYS, ndim, torch.int32))
    qty = _ints(g, 1, 51, n, torch.int32).double()
    price, disc = _measures(g, qty)
    fact = dict(fk=_ints(g, 0, ndim, n, torch.int32), flag=_ints(g, 0, 3, n, torch.int8),
                status=_ints(g, 0, 2, n, torch.int8), qty=qty, price=price, disc=disc)
    return dim, fact


@functools.lru_cache(maxsize=4)
def _zipf_cdf(ranks, s):
    return torch.from_numpy(D.zipf_cdf(ranks, s)).to(DEV)


def _zipf(g, n, ranks, dtype, s=1.1):
    """Keys 1..ranks with Zipf(s) counts, each at least once (so that the
    number of groups is the same for every seed)."""
    cdf = _zipf_cdf(ranks, s)
    key = torch.empty(n, device=DEV, dtype=dtype)
    for i in range(0, n, 1 << 25):
        m = min(1 << 25, n - i)
        u = torch.rand(m, generator=g, device=DEV, dtype=torch.float64)
        key[i:i + m] = (torch.searchsorted(cdf, u, right=True) + 1).clamp_(max=ranks).to(dtype)
    some = torch.randperm(n, generator=g, device=DEV, dtype=torch.int32)[:ranks].long()
    key[some] = torch.arange(1, ranks + 1, device=DEV, dtype=dtype)
    return key


def _tables(case, seed):
    """The columns a case's query reads, as torch tensors by table."""
    g, kind = _gen(seed), case["kind"]
    if kind in ("filter_agg", "filter_fused"):
        return dict(line=_line(g, case["rows"]))
    if kind == "join_group":
        dim, fact = _join(g, case["rows"], case["dim"])
        return dict(dim=dim, fact=fact)
    if kind in ("group_agg", "order_pair"):
        n = case["rows"]
        t = dict(key=_zipf(g, n, case["ranks"], torch.int32 if case["key"] == "i32" else torch.int64))
        if kind == "group_agg":
            t["payload"] = _uniform(g, 0.0, 1e5, n)
        else:
            t["sec"] = _ints(g, 0, 2 ** 20 + 1, n, torch.int32)
        return dict(order=t)
    if kind == "order_top":
        n = case["rows"]
        revenue = torch.round(_uniform(g, 9.0, 5.0e5, n) * 1e4) / 1e4
        return dict(order=dict(revenue=revenue, date=_ints(g, D.DAYS0, D.DAYS0 + D.NDAYS, n, torch.int32),
                               key=torch.randperm(n, generator=g, device=DEV, dtype=torch.int32)))
    if kind == "semi_join":
        # a fixed share of the rows finds its key in the set (so that the
        # selection has the same length for every seed)
        n, d = case["rows"], case["dim"]
        dim = torch.randperm(d, generator=g, device=DEV, dtype=torch.int32)
        k = max(2, int(d * 365 / D.NDAYS))
        at = _ints(g, k, d, n, torch.int32)
        hits = torch.randperm(n, generator=g, device=DEV, dtype=torch.int32)[:int(n * 365 / D.NDAYS)].long()
        at[hits] = _ints(g, 0, k, hits.numel(), torch.int32)
        qty = _ints(g, 1, 51, n, torch.int32)
        return dict(keep=dict(pk=dim[:k].clone()), fact=dict(fk=dim[at.long()], price=_measures(g, qty)[0]))
    if kind == "batch":
        t = {}
        for p, n in enumerate(B.log_uniform_sizes(case["plans"], case["lo"], case["hi"])):
            t["dim%d" % p], t["fact%d" % p] = _join(g, int(n), max(2, int(n) // 4))
        return t
    dim, fact = _join(g, case["rows"], case["dim"])
    return dict(line=_line(g, case["line"]), dim=dim, fact=fact,
                order=dict(key=_zipf(g, case["order"], max(1000, case["order"] // 15), torch.int64),
                           sec=_ints(g, 0, 2 ** 20 + 1, case["order"], torch.int32)))


# ------------------------------------------------------- vectors in and out
_TYP = {torch.int8: H_C, torch.int32: H_I, torch.int64: H_L, torch.float64: H_E}
_STR = {H_B: ("|b1", torch.bool), H_C: ("|i1", torch.int8), H_I: ("<i4", torch.int32), H_L: ("<i8", torch.int64),
        H_E: ("<f8", torch.float64)}


def _node(t):
    """A vector node over a tensor's memory."""
    v = V0()
    v.typ, v.len, v.g = _TYP[t.dtype], t.numel(), t.data_ptr()
    return v


class _View:
    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=3)


def _tensor(v, n=None, g=None):
    """A result vector as a tensor over its memory (a number when it has one element)."""
    n = v.len if n is None else n
    typestr, dtype = _STR[v.typ]
    if n == 0:
        return torch.empty(0, dtype=dtype, device=DEV)
    if n == 1:
        return {H_B: v.b, H_C: v.j, H_I: v.i32, H_L: v.i64, H_E: v.f64}[v.typ]
    return torch.as_tensor(_View(v.g if g is None else g, n, typestr), device=DEV)


def _row_lists(vals, n):
    """The concatenated row lists of a @group result: its values point into one i64 vector."""
    before = 0
    for i in range(vals.len):
        v = V0.from_address(vals.g + 32 * i)
        if v.len > 1:
            return torch.as_tensor(_View(v.g - 8 * before, n, "<i8"), device=DEV)
        before += v.len
    raise ValueError("every group has one row")


@functools.lru_cache(maxsize=None)
def _chain(lo, hi):
    return P.Chain(horsepower_gb300.load(), P.Q6_CHAIN.format(lo=lo, hi=hi))


_RESULT = np.dtype(dict(names=["ngroups", "flag", "st", "sum_qty", "avg_price", "sum_disc", "count"],
                        formats=["<i8", ("i1", B.MAXG), ("i1", B.MAXG), ("<f8", B.MAXG), ("<f8", B.MAXG),
                                 ("<f8", B.MAXG), ("<i8", B.MAXG)],
                        offsets=[getattr(B.Result, f).offset for f in
                                 ("ngroups", "flag", "st", "sum_qty", "avg_price", "sum_disc", "count")],
                        itemsize=C.sizeof(B.Result)))


# ------------------------------------------------------------------ prepare
class State:
    """A query's tables as nodes, and what its program keeps beside them."""

    def __init__(self, case, seed):
        L = self.L = horsepower_gb300.load()
        self.case, self.tensors = case, _tables(case, seed)
        torch.cuda.synchronize()
        for name, cols in self.tensors.items():
            setattr(self, name, {k: _node(t) for k, t in cols.items()})
        kind = case["kind"]
        if kind == "filter_fused":
            self.chain = _chain(D.WIN_LO, D.WIN_HI)
        elif kind == "batch":
            n = case["plans"]
            los = [D.DAYS0 + (p * 131) % (D.NDAYS - 365) for p in range(n)]
            self.plans = (B.Plan * n)(*[B.make_plan(getattr(self, "dim%d" % p), getattr(self, "fact%d" % p),
                                                    los[p], los[p] + 365) for p in range(n)])
            self.results = (B.Result * n)()
            L.lib.hgpuBatchJoinGroup.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p]
        elif kind == "serve":
            n = case["requests"]
            self.requests = S.request_stream(n, 0, seed, key_hi=max(1000, case["order"] // 15))
            self.server = S.Server(L, self.line, self.dim, self.fact, self.order)
            self.arr = (S.Request * n)(*self.requests)
            self.out, self.results = (S.Response * n)(), (B.Result * n)()
            self.rows = np.zeros((n, S.TOPK), np.int64)
            for i in range(n):
                self.out[i].group = C.pointer(self.results[i])
                self.out[i].rows = C.cast(self.rows.ctypes.data + 8 * S.TOPK * i, C.POINTER(C.c_longlong))
            self.stats = S.Stats()
        self.heap = L.lib.getHeapOffset()

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()


def prepare(case, seed):
    return State(case, seed)


# ---------------------------------------------------------------------- run
def run(s):
    L = s.L
    L.free_inputs()
    L.lib.setHeapOffset(s.heap)
    return _RUN[s.case["kind"]](L, s)


def _run_filter_agg(L, s):
    return [_tensor(P.filter_aggregate(L, s.line))]


def _run_filter_fused(L, s):
    return [_tensor(P.filter_aggregate_fused(L, s.line, s.chain))]


def _run_join_group(L, s):
    return [_tensor(v) for v in P.join_group_compiled(L, s.dim, s.fact)]


def _run_group_agg(L, s):
    g = L.call("pfnGroup", s.order["key"])
    vals = L.call("pfnValues", g)
    keys = L.call("pfnKeys", g)
    sums = P.group_agg(L, "pfnSum", s.order["payload"], vals)
    counts = P.group_agg(L, "pfnLen", s.order["payload"], vals)
    return [_tensor(keys), _row_lists(vals, s.order["key"].len), _tensor(sums), _tensor(counts)]


def _run_order_pair(L, s):
    dirs = L.vec(np.array([True, True]), H_B)
    return [_tensor(L.call("pfnOrderBy", L.list([s.order["key"], s.order["sec"]]), dirs))]


def _run_order_top(L, s):
    o = s.order
    dirs = L.vec(np.array([False, True]), H_B)
    perm = L.call("pfnOrderBy", L.list([o["revenue"], o["date"]]), dirs)
    cols = P.index_many(L, [o["key"], o["revenue"], o["date"]], perm)
    return [_tensor(perm)] + [_tensor(v) for v in cols]


def _run_semi_join(L, s):
    mask = L.call("pfnMember", s.fact["fk"], s.keep["pk"])
    price = L.call("pfnCompress", mask, s.fact["price"])
    stats = [L.call(f, price) for f in ("pfnAvg", "pfnMin", "pfnMax")]
    return [_tensor(mask), _tensor(price)] + [_tensor(v) for v in stats]


def _results(results, n):
    r = np.frombuffer(results, _RESULT, n)
    return [r[k] for k in _RESULT.names]


def _run_batch(L, s):
    n = s.case["plans"]
    rc = L.lib.hgpuBatchJoinGroup(s.plans, n, s.results)
    if rc:
        raise RuntimeError("hgpuBatchJoinGroup: %d" % rc)
    return _results(s.results, n)


def _run_serve(L, s):
    n = s.case["requests"]
    rc = L.lib.hgpuServerRun(s.server.h, s.arr, n, s.out, S.BATCHED, C.byref(s.stats))
    if rc:
        raise RuntimeError("hgpuServerRun: %d" % rc)
    return [np.array([o.value for o in s.out]), s.rows, np.array([o.nrows for o in s.out])] + _results(s.results, n)


_RUN = {k[5:]: f for k, f in list(globals().items()) if k.startswith("_run_")}


# --------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once, at element width; a column
    read through a selection counts its selected rows.  One compare, add or
    multiply per row and statement."""
    kind = case["kind"]
    sel = 365 / D.NDAYS
    if kind in ("filter_agg", "filter_fused"):
        return dict(bytes=24 * case["rows"], flops=8 * case["rows"])
    if kind == "join_group":
        n, d = case["rows"], case["dim"]
        return dict(bytes=int(4 * d + 4 * d * sel + 4 * n + 26 * n * sel), flops=int(2 * d + n + 3 * n * sel))
    if kind == "group_agg":
        n, w = case["rows"], 4 if case["key"] == "i32" else 8
        groups = min(case["ranks"], n)
        return dict(bytes=(w + 8 + 8) * n + 24 * groups, flops=n)
    if kind == "order_pair":
        n, w = case["rows"], 4 if case["key"] == "i32" else 8
        return dict(bytes=(w + 4 + 8) * n, flops=n)
    if kind == "order_top":
        n = case["rows"]
        return dict(bytes=(12 + 8) * n + (8 + 16 + 16) * n, flops=n)
    if kind == "semi_join":
        n, k = case["rows"], int(case["dim"] * sel)
        return dict(bytes=int(5 * n + 4 * k + 16 * n * sel), flops=int(n + 3 * n * sel))
    if kind == "batch":
        sizes = [int(v) for v in B.log_uniform_sizes(case["plans"], case["lo"], case["hi"])]
        parts = [work(dict(kind="join_group", rows=n, dim=max(2, n // 4))) for n in sizes]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    # serve: every table once, whatever the number of requests that share it
    n = case["requests"]
    return dict(bytes=24 * case["line"] + 8 * case["dim"] + 30 * case["rows"] + 8 * case["order"],
                flops=int(0.6 * n * 8 * case["line"] + 0.3 * n * 4 * case["rows"] * sel + case["order"]))


# -------------------------------------------------------------------- exact
def _q6(t, lo, hi):
    m = (t["shipdate"] >= lo) & (t["shipdate"] < hi) & (t["qty"] < 24) & (t["disc"] >= 0.05) & (t["disc"] <= 0.07)
    return float((t["price"][m] * t["disc"][m]).sum())


def _join_group_sums(dim, fact, lo, hi):
    """Per group in ascending (flag, status) order: sum(qty), avg(price), sum(disc)."""
    keep = torch.zeros(dim["pk"].numel(), dtype=torch.bool, device=DEV)
    keep[dim["pk"].long()] = (dim["date"] >= lo) & (dim["date"] < hi)
    m = keep[fact["fk"].long()]
    code = (fact["flag"][m].long() << 8) | fact["status"][m].long()
    codes = torch.unique(code)
    cols = [[], [], []]
    for c in codes.tolist():
        at = code == c
        for k, (name, agg) in enumerate((("qty", torch.sum), ("price", torch.mean), ("disc", torch.sum))):
            cols[k].append(float(agg(fact[name][m][at])))
    return [np.array(v) for v in cols]


def _padded(parts, n):
    out = [np.zeros((n, B.MAXG)) for _ in range(3)]
    for i, sums in parts.items():
        for k in range(3):
            out[k][i, :len(sums[k])] = sums[k]
    return [None, None, None] + out + [None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "order_pair":
        return None
    t = _tables(case, seed)
    if kind in ("filter_agg", "filter_fused"):
        return [_q6(t["line"], D.WIN_LO, D.WIN_HI)]
    if kind == "join_group":
        return [None, None] + _join_group_sums(t["dim"], t["fact"], D.WIN_LO, D.WIN_HI) + [None]
    if kind == "group_agg":
        key, inv = torch.unique(t["order"]["key"], return_inverse=True)
        sums = torch.zeros(key.numel(), dtype=torch.float64, device=DEV)
        sums.index_add_(0, inv, t["order"]["payload"])
        return [None, None, sums, None]
    if kind == "order_top":
        o = t["order"]
        return [None, None, torch.sort(o["revenue"], descending=True).values, None]
    if kind == "semi_join":
        keep = torch.zeros(case["dim"], dtype=torch.bool, device=DEV)
        keep[t["keep"]["pk"].long()] = True
        price = t["fact"]["price"][keep[t["fact"]["fk"].long()]]
        return [None, price, float(price.mean()), float(price.min()), float(price.max())]
    if kind == "batch":
        n = case["plans"]
        los = [D.DAYS0 + (p * 131) % (D.NDAYS - 365) for p in range(n)]
        return _padded({p: _join_group_sums(t["dim%d" % p], t["fact%d" % p], los[p], los[p] + 365)
                        for p in range(n)}, n)
    n = case["requests"]
    reqs = S.request_stream(n, 0, seed, key_hi=max(1000, case["order"] // 15))
    value = np.array([_q6(t["line"], r.lo, r.hi) if r.kind == S.FILTER_AGG else 0.0 for r in reqs])
    joins = {i: _join_group_sums(t["dim"], t["fact"], r.lo, r.hi) for i, r in enumerate(reqs) if r.kind == S.JOIN_GROUP}
    return [value, None, None] + _padded(joins, n)
