"""The groupbys that are timed: what users of this package call, from a lookup
of two thousand rows to the 100M-row workloads of `bench.py`.

A case names the entry point (`call`), the rows and distinct keys, how the keys
are drawn, and the value columns with their aggregations.  `run` makes one call
(or one batch, or one burst of served queries) and hands the groups back in key
order, as a program that joins, prints or stores them wants them: the engine's
own group order is arbitrary.
"""
import math

import numpy as np
import torch

import cudf_b200 as cb
from cudf_b200 import aggregation as agg

_WIDTH = {"i64": 8, "i32": 4, "i16": 2, "i8": 1, "u8": 1, "f64": 8, "f32": 4, "bool": 1}
_SPAN = 1 << 20  # values of a second key column stay below this


def listed():
    every = "sum,count,min,max,mean"
    return [
        # a lookup table or one dashboard tile: nothing but launches and latency
        dict(name="tile_2k", call="groupby", rows=2_000, groups=50, keys="i32", dist="uniform", key_nulls=0.0,
             nulls=0.0, offset=0, requests="i64=sum,count,min,max f64=mean"),
        # a small table with nulls and many groups, the smallest queries of a serving stream
        dict(name="table_50k", call="groupby", rows=50_021, groups=5_000, keys="i64", dist="uniform", key_nulls=0.0,
             nulls=0.1, offset=0, requests="i64=sum,count,mean f64=sum,count,mean"),
        # bench.py --workload small
        dict(name="report_1M", call="groupby", rows=1_000_000, groups=1_000, keys="i32", dist="uniform",
             key_nulls=0.0, nulls=0.0, offset=0, requests="i64=sum,count,min,max f64=mean"),
        # the mean query of bench.py's serving stream, run alone
        dict(name="query_2M6", call="groupby", rows=2_611_199, groups=30_000, keys="i64", dist="uniform",
             key_nulls=0.0, nulls=0.1, offset=0, requests="i64=sum,count,mean f64=sum,count,mean"),
        # DataFrame.groupby(...).agg(...) with a spread statistic, sorted by key as pandas does it
        dict(name="frame_var_4M", call="frame", rows=4_000_037, groups=20_000, keys="i64", dist="uniform",
             key_nulls=0.0, nulls=0.0, offset=0, requests="f64=mean,var,std i64=sum,min,max"),
        # a pricing summary: two code columns, six groups, every row contends for them
        dict(name="codes_60M", call="groupby", rows=60_000_000, groups=6, keys="i8,i8", dist="uniform",
             key_nulls=0.0, nulls=0.0, offset=0, requests="f64=sum,mean f64=sum,mean i32=sum,count"),
        # a slice of a wide table: narrow types, an offset that no vector load is aligned to
        dict(name="slice_20M", call="groupby", rows=20_000_003, groups=100_000, keys="i32", dist="uniform",
             key_nulls=0.05, nulls=0.1, offset=3, requests="f32=sum,min,max i16=sum,max u8=sum,count"),
        # bench.py's default line
        dict(name="rows_100M", call="groupby", rows=100_000_000, groups=1_000_000, keys="i64", dist="uniform",
             key_nulls=0.0, nulls=0.1, offset=0, requests=f"i64={every} f64={every} f32={every}"),
        # bench.py --workload zipf: two key columns, skew, null keys as groups
        dict(name="zipf_100M", call="groupby", rows=100_000_000, groups=50_000_000, keys="i32,i64", dist="zipf",
             key_nulls=0.05, nulls=0.0, offset=0, requests="i64=sum,count,max f64=sum,count,max"),
        # deduplication: nearly as many groups as rows
        dict(name="dedup_40M", call="groupby", rows=40_000_000, groups=40_000_000, keys="i64", dist="uniform",
             key_nulls=0.0, nulls=0.0, offset=0, requests="f32=sum,count i32=max"),
        # bench.py --workload batch: independent instances in one launch, replayed as a graph
        dict(name="batch_12", call="batch", rows=12_000_000, groups=20_000, keys="i32", dist="uniform", parts=12,
             key_nulls=0.0, nulls=0.05, offset=0, requests="i64=sum,count f64=sum,min,max,mean"),
        # bench.py --workload serve: a burst of queries of mixed sizes
        dict(name="serve_12", call="serve", rows=16_000_000, groups=100_000, keys="i64", dist="uniform", parts=12,
             key_nulls=0.0, nulls=0.1, offset=0, requests="i64=sum,count,mean f64=sum,mean"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["groupby"] * 8 + ["frame", "frame", "batch", "serve"])
    dist, keys, key_nulls, nulls, offset = "uniform", "i64", 0.0, rng.choice([0.0, 0.1]), 0
    case = dict(call=call)
    if call == "groupby":
        rows = _log(rng, 1_000, 60_000_000) | 1
        keys = rng.choice(["i64", "i64", "i32", "i32,i64", "f64", "i8,i8"])
        groups = 6 if keys == "i8,i8" else min(_log(rng, 4, 2 * rows), 40_000_000)
        if keys == "i32,i64" and rng.random() < 0.5:
            dist, groups = "zipf", max(groups, 10_000)
        if keys in ("i32", "i32,i64"):
            key_nulls = rng.choice([0.0, 0.05])
        if keys in ("i64", "i32"):
            offset = rng.choice([0, 0, 1, 13, 32])
        requests = rng.choice([
            "i64=sum,count,min,max f64=mean", "i64=sum,count,mean f64=sum,count,mean",
            "i64=sum,count,min,max,mean f64=sum,count,min,max,mean f32=sum,count,min,max,mean",
            "f32=sum,min,max i16=sum,max u8=sum,count", "f64=sum,mean i32=sum,count", "bool=sum,count i32=min,max",
            "f64=argmin,argmax i32=argmax", "f32=sum,count i8=min"])
    elif call == "frame":
        rows = _log(rng, 10_000, 20_000_000) | 1
        groups = _log(rng, 10, min(rows, 200_000))
        keys, nulls = rng.choice(["i64", "i32"]), 0.0
        requests = rng.choice(["f64=mean,var,std i64=sum,min,max", "f64=sum,mean f32=std", "i32=sum,count,mean"])
    else:
        rows = _log(rng, 100_000, 16_000_000)
        groups = _log(rng, 10, 100_000)
        keys = "i32" if call == "batch" else "i64"
        requests = "i64=sum,count f64=sum,min,max,mean" if call == "batch" else "i64=sum,count,mean f64=sum,mean"
        case["parts"] = rng.randint(4, 12)
    case.update(rows=rows, groups=groups, keys=keys, dist=dist, key_nulls=key_nulls, nulls=nulls, offset=offset,
                requests=requests)
    return case


# -- inputs -------------------------------------------------------------------
def _requests(case):
    return [(r.split("=")[0], r.split("=")[1].split(",")) for r in case["requests"].split()]


def _aggregation(name):
    return {"sum": agg.sum, "count": agg.count, "min": agg.min, "max": agg.max, "mean": agg.mean,
            "var": lambda: agg.variance(1), "std": lambda: agg.std(1), "argmin": agg.argmin,
            "argmax": agg.argmax}[name]()


def _value(kind, n, g):
    dev = g.device
    if kind == "i64":
        return torch.randint(-10**9, 10**9 + 1, (n,), device=dev, generator=g, dtype=torch.int64)
    if kind == "i32":
        return torch.randint(-10**6, 10**6 + 1, (n,), device=dev, generator=g, dtype=torch.int32)
    if kind == "i16":
        return torch.randint(-30_000, 30_001, (n,), device=dev, generator=g, dtype=torch.int16)
    if kind == "i8":
        return torch.randint(-128, 128, (n,), device=dev, generator=g, dtype=torch.int8)
    if kind == "u8":
        return torch.randint(0, 256, (n,), device=dev, generator=g, dtype=torch.uint8)
    if kind == "bool":
        return torch.randint(0, 2, (n,), device=dev, generator=g, dtype=torch.uint8).to(torch.bool)
    if kind == "f64":
        return torch.randn(n, device=dev, generator=g, dtype=torch.float64)
    return torch.empty(n, device=dev, dtype=torch.float32).log_normal_(0.0, 1.0, generator=g)


def _ids(case, groups, n, g):
    if case["dist"] == "uniform":
        return torch.randint(0, groups, (n,), device=g.device, generator=g)
    # P(p) proportional to (p + 1)^-1.1 on [0, groups): inverse of the continuous distribution
    u = torch.rand(n, device=g.device, generator=g, dtype=torch.float64)
    top = (groups + 1.0) ** -0.1
    return ((1.0 - u * (1.0 - top)) ** -10.0 - 1.0).to(torch.int64).clamp_(0, groups - 1)


def _tensors(case, rows, groups, g):
    """([key tensor, valid or None] per key column, [value tensor, valid or None] per request).

    Which group a row belongs to, and which keys are null, is drawn once per shape and turned by a
    number of rows of the seed's own, so that every seed has the same number of groups; keys and
    values are the seed's."""
    n = rows + case["offset"]
    fixed = torch.Generator(device=g.device)
    fixed.manual_seed(rows * 31 + groups)
    turn, base = (int(t) for t in torch.randint(0, 1000, (2,), device=g.device, generator=g))
    turn = turn * rows // 1000

    def turned(t):  # the sliced-off rows ahead of the offset stay outside
        t[case["offset"]:] = torch.roll(t[case["offset"]:], turn)
        return t

    ids = turned(_ids(case, groups, n, fixed))
    kinds = case["keys"]
    if kinds == "i64":
        table = torch.randint(-2**62, 2**62, (groups,), device=g.device, generator=g, dtype=torch.int64)
        keys = [table[ids]]
    elif kinds == "i32":
        keys = [(ids + base).to(torch.int32)]
    elif kinds == "f64":
        keys = [ids.to(torch.float64) * 0.25 - base]
    elif kinds == "i8,i8":
        keys = [(torch.div(ids, 2, rounding_mode="floor") + base % 100).to(torch.int8), (ids % 2).to(torch.int8)]
    else:
        keys = [(torch.div(ids, 1000, rounding_mode="floor") + base).to(torch.int32), ids % 1000]
    del ids

    def some(share, gen):
        return torch.rand(n, device=g.device, generator=gen) >= share if share else None

    def key_valid():
        v = some(case["key_nulls"], fixed)
        return None if v is None else turned(v)

    return ([(k, key_valid()) for k in keys],
            [(_value(kind, n, g), some(case["nulls"], g)) for kind, _ in _requests(case)])


def _parts(case, seed):
    """Rows and distinct keys of the instances of a batch or of the queries of a burst: spread over their logarithm."""
    if "parts" not in case:
        return [(case["rows"], case["groups"])]
    r = np.random.default_rng(len(case["requests"]) + case["parts"])
    share = np.exp(r.uniform(np.log(0.01), 0.0, case["parts"]))
    share /= share.sum()
    groups = np.exp(r.uniform(np.log(4), np.log(max(5, case["groups"])), case["parts"]))
    return [(max(1000, int(case["rows"] * s)), int(max(1, c))) for s, c in zip(share, groups)]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _column(t, valid, case, rows):
    c = cb.Column.from_tensor(t, valid)
    return cb.Column(c.type_id, c.data, c.mask, size=rows, offset=case["offset"])


_SERVER = []


def _server():
    if not _SERVER:
        _SERVER.append(cb.Server(memory_cap_bytes=150 << 30))
    return _SERVER[0]


def prepare(case, seed):
    g = _generator(seed)
    queries = []
    for rows, groups in _parts(case, seed):
        keys, values = _tensors(case, rows, groups, g)
        kt = cb.Table([_column(t, v, case, rows) for t, v in keys])
        cols = [_column(t, v, case, rows) for t, v in values]
        queries.append((kt, [cb.GroupByRequest(c, [_aggregation(a) for a in aggs])
                             for c, (_, aggs) in zip(cols, _requests(case))]))
    state = {"case": case, "queries": queries,
             "policy": cb.NullPolicy.INCLUDE if case["keys"] == "i32,i64" else cb.NullPolicy.EXCLUDE}
    if case["call"] == "frame":
        kt, reqs = queries[0]
        state["frame"] = cb.DataFrame({"k": kt[0], **{f"v{i}": r.values for i, r in enumerate(reqs)}})
        state["spec"] = {f"v{i}": aggs for i, (_, aggs) in enumerate(_requests(case))}
    elif case["call"] == "batch":
        state["batch"] = cb.BatchGroupBy(queries, use_graph=True)
    elif case["call"] == "serve":
        state["server"] = _server()
    return state


# -- one pass -----------------------------------------------------------------
def _code(columns):
    """One sortable tensor for the key columns: a null comes first."""
    if len(columns) == 1 and columns[0][1] is None:
        return columns[0][0]
    code = None
    for t, valid in columns:
        c = t.to(torch.int64) + 1
        if valid is not None:
            c = torch.where(valid, c, torch.zeros_like(c))
        code = c if code is None else code * _SPAN + c
    return code


def _in_key_order(keys, results):
    """The key and result columns of one or several groupbys, ordered by (groupby, key)."""
    codes = [_code([(c.data, c.valid() if c.mask is not None else None) for c in k]) for k in keys]
    columns = [[*k, *(c for t in r for c in t)] for k, r in zip(keys, results)]
    if len(codes) == 1:
        order = torch.argsort(codes[0])
        out = [c.data.index_select(0, order) for c in columns[0]]
    else:  # one gather per column for all of them
        at, begin = [], 0
        for c in codes:
            at.append(torch.argsort(c) + begin)
            begin += c.numel()
        order = torch.cat(at)
        out = [torch.cat([c.data for c in same]).index_select(0, order) for same in zip(*columns)]
    return {"columns": out, "nulls": [sum(c.null_count for c in same) for same in zip(*columns)],
            "groups": [c.numel() for c in codes]}


def run(state):
    call = state["case"]["call"]
    if call == "groupby":
        kt, reqs = state["queries"][0]
        keys, results = cb.GroupBy(kt, state["policy"]).aggregate(reqs)
        return _in_key_order([keys], [results])
    if call == "frame":
        out = state["frame"].groupby("k", sort=True).agg(state["spec"])
        return {"columns": [c.values() for _, c in out.index] + [out[name].values() for name in out.columns]}
    if call == "batch":
        batch = state["batch"]
        batch.run()
        got = [batch.result(i) for i in range(len(batch))]
        return _in_key_order([k for k, _ in got], [r for _, r in got])
    server = state["server"]
    ids = [server.submit(kt, reqs, state["policy"]) for kt, reqs in state["queries"]]
    for q in ids:
        server.wait(q)
    got = [server.result(q) for q in ids]
    out = _in_key_order([k for k, _ in got], [r for _, r in got])
    torch.cuda.current_stream().synchronize()  # the copies are made: the server may have its buffers back
    for q in ids:
        server.release(q)
    return out


# -- what a pass cannot do without --------------------------------------------
def _distinct(case, rows, groups):
    if case["dist"] == "uniform":
        return groups * -math.expm1(-rows / groups)
    p = np.exp(np.linspace(0.0, math.log(groups + 1.0), 20_001))
    mid, width = np.sqrt(p[1:] * p[:-1]), np.diff(p)
    prob = 0.1 * mid ** -1.1 / (1.0 - (groups + 1.0) ** -0.1)
    seen = float(np.sum(width * -np.expm1(-rows * prob)))
    return seen + (min(seen, 51_000) if case["key_nulls"] else 0)


def work(case):
    bytes_, ops = 0.0, 0.0
    kw = [_WIDTH[k] for k in case["keys"].split(",")]
    for rows, groups in _parts(case, 0):
        found = _distinct(case, rows, groups)
        bytes_ += rows * (sum(kw) + (len(kw) / 8 if case["key_nulls"] else 0)) + found * sum(kw)
        for kind, aggs in _requests(case):
            bytes_ += rows * (_WIDTH[kind] + (1 / 8 if case["nulls"] else 0))
            for a in aggs:
                wide = 4 if a in ("count", "argmin", "argmax") else 8 if a in ("sum", "mean", "var", "std") else _WIDTH[kind]
                bytes_ += found * (4 if a == "sum" and kind == "f32" else wide)
                ops += rows * (3 if a in ("var", "std") else 1)
    return {"bytes": bytes_, "flops": ops}


# -- the same results in 64 bits ----------------------------------------------
def _exact_one(case, rows, groups, g):
    """Per result column: float64 values in key order, or None where the result is a whole number."""
    keys, values = _tensors(case, rows, groups, g)
    o = case["offset"]
    code = _code([(t[o:], None if v is None else v[o:]) for t, v in keys])
    keep = None
    if case["keys"] != "i32,i64" and case["key_nulls"]:
        keep = keys[0][1][o:]
        code = code[keep]
    uniq, inv = torch.unique(code, return_inverse=True)
    n = uniq.numel()
    out = [None] * len(keys)
    for (t, valid), (kind, aggs) in zip(values, _requests(case)):
        t, valid = t[o:], None if valid is None else valid[o:]
        if keep is not None:
            t, valid = t[keep], None if valid is None else valid[keep]
        at = inv
        if valid is not None:
            t, at = t[valid], inv[valid]
        x = t.to(torch.float64)
        zero = torch.zeros(n, dtype=torch.float64, device=x.device)
        cnt = torch.bincount(at, minlength=n).to(torch.float64)
        total = zero.clone().index_add_(0, at, x)
        mean = total / cnt.clamp(min=1)
        is_float = kind in ("f64", "f32")
        for a in aggs:
            v = None
            if a == "sum" and is_float:
                v = total
            elif a == "mean":
                v = mean
            elif a in ("min", "max") and is_float:
                v = zero.clone().scatter_reduce_(0, at, x, "amin" if a == "min" else "amax", include_self=False)
            elif a in ("var", "std"):
                d = x - mean[at]
                v = zero.clone().index_add_(0, at, d * d) / (cnt - 1).clamp(min=1)
                v = torch.where(cnt > 1, v, zero)
                v = v.sqrt() if a == "std" else v
            out.append(v)
    return out


def exact(case, seed):
    g = _generator(seed)
    parts = [_exact_one(case, rows, groups, g) for rows, groups in _parts(case, seed)]
    columns = [None if same[0] is None else torch.cat(same) for same in zip(*parts)]
    if all(c is None for c in columns):
        return None
    if case["call"] == "frame":
        return {"columns": columns}
    return {"columns": columns, "nulls": None, "groups": None}
