"""Queries the engine is used for, from the smallest lookup to the largest roll-up, as repeatable cases.

A case is a dict of plain values. `prepare` builds what a program holds before the query (tables in the
column cache, device or host columns, the plan), `run` executes the query once through the engine's
public interface and returns its whole result, `exact` recomputes the floating-point outputs in 64 bits
with torch alone, and `work` counts the bytes a query cannot do without.

Kinds and their ranges:

  group    filter + projection + GROUP BY a small key over a cached table, result on the host: the
           dashboard query (2^12 .. 2^26 rows, 16 .. 2048 groups)
  cold     the same over host columns that are not cached, narrow types: a table's first query
           (2^12 .. 2^21 rows)
  select   filter + projection of a cached table, result left on the device, one column with NULLs or
           none (2^12 .. 2^25 rows)
  rollup   GROUP BY two keys of a cached table, skewed first key (2^20 .. 2^27 rows), and GROUP BY one
           evenly spread key of device columns (2^16 .. 2^25 rows); the caller keeps the aggregates in
           dense arrays addressed by the key
  ids      GROUP BY a sparse BIGINT id, result ordered by id (2^16 .. 2^24 rows)
  join     fact table joined to a build side with unique keys, grouped by a build column
           (2^18 .. 2^28 probe rows, 2^12 .. 2^24 build rows)
  star     fact table joined to a dimension, filtered and projected, rows left on the device
           (2^16 .. 2^25 fact rows)
  pairs    a join whose right keys repeat, its pairs left on the device (2^14 .. 2^22 left rows)
  batch    many small dashboard queries in one call (4 .. 20 queries, 2^10 .. 2^22 rows each)
"""
from __future__ import annotations

import itertools
import math
import random

import numpy as np
import torch

from vectisdb_b200.engine import (ColumnCache, ExecuteOptions, GpuAggregateKind as A, GpuColumn, GpuEngine,
                                  GpuTableRef, GpuValueType as T, make_aggregate, make_column, make_device_column,
                                  make_expr, make_filter, make_group_by, make_join, make_projection, make_scan)
from vectisdb_b200.workloads import c0_plan, c1_plan, c2_plan, cp_plan

DEV = "cuda"
TS_MID = 1 << 61       # the timestamps are uniform over [0, 2^62)
ROLLUP_B = 16          # second key of the skewed roll-up
JOIN_GROUPS = 4096


# ---- cases ---------------------------------------------------------------------------------------------


def listed():
    return [
        # a dashboard tile over a small table: the latency of one call
        {"name": "group_4k", "kind": "group", "rows": 4096, "groups": 16},
        # the filter + group-by benchmark configuration
        {"name": "group_16m", "kind": "group", "rows": 1 << 24, "groups": 1024},
        # the first query over a table that is not cached yet; narrow column types
        {"name": "cold_2m", "kind": "cold", "rows": 2_097_143, "groups": 300},
        # the filter + projection benchmark configuration
        {"name": "select_16m", "kind": "select", "rows": 1 << 24, "nulls": False},
        # the same query over a ragged table whose measure has NULLs
        {"name": "select_nulls_3m", "kind": "select", "rows": 3_000_017, "nulls": True},
        # the high-cardinality group-by benchmark configuration: the largest roll-up
        {"name": "rollup_skew_128m", "kind": "rollup", "rows": 1 << 27, "keys": 1 << 20, "skew": True},
        # a roll-up by an evenly spread key of columns another program left on the device
        {"name": "rollup_even_10m", "kind": "rollup", "rows": 10_000_019, "keys": 1_000_003, "skew": False},
        # totals per BIGINT user id
        {"name": "ids_8m", "kind": "ids", "rows": 8_000_009, "keys": 600_011},
        # the join + group-by benchmark configuration, both sides device columns
        {"name": "join_256m", "kind": "join", "rows": 1 << 28, "build": 1 << 24},
        # a fact table against a dimension, row by row
        {"name": "star_6m", "kind": "star", "rows": 6_000_003, "build": 200_003},
        # a many-to-many join, every pair kept
        {"name": "pairs_4m", "kind": "pairs", "rows": 4_000_037, "build": 1_000_003, "keys": 500_009},
        # a screen of dashboard tiles, each over its own table
        {"name": "batch_20", "kind": "batch", "queries": 20, "mix": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["group", "group", "cold", "select", "select", "rollup", "rollup", "ids", "join", "join",
                       "star", "pairs", "batch"])
    if kind == "group":
        return {"kind": kind, "rows": _log(rng, 1 << 12, 1 << 26), "groups": _log(rng, 16, 2048)}
    if kind == "cold":
        return {"kind": kind, "rows": _log(rng, 1 << 12, 1 << 21), "groups": _log(rng, 16, 1000)}
    if kind == "select":
        return {"kind": kind, "rows": _log(rng, 1 << 12, 1 << 25), "nulls": rng.random() < 0.5}
    if kind == "rollup":
        if rng.random() < 0.5:
            return {"kind": kind, "rows": _log(rng, 1 << 20, 1 << 27), "keys": _log(rng, 1 << 12, 1 << 20),
                    "skew": True}
        rows = _log(rng, 1 << 16, 1 << 25)
        return {"kind": kind, "rows": rows, "keys": _log(rng, 1 << 13, min(rows // 2, 1 << 23)), "skew": False}
    if kind == "ids":
        rows = _log(rng, 1 << 16, 1 << 24)
        return {"kind": kind, "rows": rows, "keys": _log(rng, 1 << 10, min(rows // 4, 1 << 20))}
    if kind == "join":
        rows = _log(rng, 1 << 18, 1 << 28)
        return {"kind": kind, "rows": rows, "build": _log(rng, 1 << 12, min(rows // 4, 1 << 24))}
    if kind == "star":
        rows = _log(rng, 1 << 16, 1 << 25)
        return {"kind": kind, "rows": rows, "build": _log(rng, 1 << 10, min(rows // 4, 1 << 22))}
    if kind == "pairs":
        rows = _log(rng, 1 << 14, 1 << 22)
        build = _log(rng, 1 << 12, 1 << 20)
        return {"kind": kind, "rows": rows, "build": build, "keys": max(16, int(build / rng.uniform(1.2, 3.0)))}
    return {"kind": kind, "queries": rng.randint(4, 20), "mix": rng.randint(100, 100000)}


# ---- inputs --------------------------------------------------------------------------------------------


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1009 + salt)
    return g


def _ints(g, n, lo, hi, dtype):
    return torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=dtype)


def _doubles(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _zipf(g, n, values, s):
    """Ranks in [0, values), rank r with a weight of about (r + 1)^-s (the continuous law, inverted), as int64."""
    e = 1.0 - s
    u = _doubles(g, n).mul_((values + 1.0) ** e - 1.0).add_(1.0)
    return u.pow_(1.0 / e).long().sub_(1).clamp_(0, values - 1)


def _spread(ids):
    """Distinct sparse 50-bit ids from small ones (an odd multiplier is a bijection modulo 2^50)."""
    return (ids * 2862933555777941757 + 3037000493) & ((1 << 50) - 1)


def _batch_shapes(case):
    rng = random.Random(case["mix"])
    shapes = []
    for _ in range(case["queries"]):
        shapes.append((_log(rng, 1 << 10, 1 << 22), _log(rng, 16, 1 << 16), round(rng.uniform(0.1, 0.9), 6),
                       rng.randint(2, 16)))
    return shapes


# How many rows a filter keeps, and how many groups have rows, depends on the sizes alone, not on the seed:
# a random order of the rows decides which of them are kept and which key each has.


def _dash_inputs(g, rows, groups, v_lt, w_mod, null_share=0.0):
    """Rows kept by v < v_lt and w % w_mod <> 0, rows that fail only the second, rows that fail the first."""
    order = torch.randperm(rows, generator=g, device=DEV)
    below = int(rows * v_lt)
    kept = below - below // w_mod
    u, w = _doubles(g, rows), _ints(g, rows, 0, 1_000_000 // w_mod, torch.int64).mul_(w_mod)
    rest = _ints(g, rows, 1, w_mod, torch.int64)
    w += torch.where(order < kept, rest, torch.where(order < below, 0, rest - 1))
    cols = {"k": (order % groups).to(torch.int32), "v": torch.where(order < below, u * v_lt, v_lt + u * (1.0 - v_lt)),
            "w": w}
    if null_share:
        cols["v_valid"] = order >= int(rows * null_share)
    return cols


def _inputs(case, seed):
    """The case's columns as device tensors, from the seed alone."""
    g, n, kind = _gen(seed), case.get("rows", 0), case["kind"]
    if kind == "group":
        return _dash_inputs(g, n, case["groups"], 0.5, 7)
    if kind == "cold":
        order = torch.randperm(n, generator=g, device=DEV)
        return {"region": (order % case["groups"] - 5).to(torch.int16), "open": order < int(0.7 * n),
                "qty": _ints(g, n, 1, 5000, torch.int32),
                "price": torch.rand(n, generator=g, device=DEV, dtype=torch.float32) * 100}
    if kind == "select":
        return _dash_inputs(g, n, 1024, 0.5, 7, 0.1 if case["nulls"] else 0.0)
    if kind == "rollup" and case["skew"]:
        return {"a": _zipf(g, n, case["keys"], 1.1).to(torch.int32), "b": _ints(g, n, 0, ROLLUP_B, torch.int32),
                "amt": _ints(g, n, 0, 1_000_000, torch.int64), "v": _doubles(g, n),
                "ts": _ints(g, n, 0, 1 << 62, torch.int64)}
    if kind == "rollup":
        return {"a": _ints(g, n, 0, case["keys"], torch.int32), "v": _doubles(g, n)}
    if kind == "ids":
        ids = _ints(g, n, 0, case["keys"], torch.int64)
        order = torch.randperm(n, generator=g, device=DEV)[: case["keys"]]
        ids[order] = torch.arange(case["keys"], device=DEV)  # every id has a row
        return {"id": _spread(ids), "v": _doubles(g, n)}
    if kind == "join":
        build, groups = case["build"], min(case["build"], JOIN_GROUPS)
        bkey = torch.randperm(build, generator=g, device=DEV)
        pkey = bkey[_zipf(g, n, build, 0.8)]
        miss = torch.rand(n, generator=g, device=DEV) < 0.1
        pkey = torch.where(miss, _ints(g, n, build, 2 * build, torch.int64), pkey)
        pkey[:groups] = bkey[:groups]  # every group has a row
        del miss
        return {"pkey": pkey, "x": _doubles(g, n), "bkey": bkey,
                "g": (torch.arange(build, device=DEV) % groups).to(torch.int32)}
    if kind == "star":
        build = case["build"]
        low = build * 6 // 10  # the dimension rows the filter keeps, and three kinds of fact rows
        dk = torch.randperm(build, generator=g, device=DEV).to(torch.int32)
        cat = _ints(g, build, 0, 600, torch.int32)
        cat[low:] = _ints(g, build - low, 600, 1000, torch.int32)
        order = torch.randperm(n, generator=g, device=DEV)
        u = _doubles(g, n)
        row = torch.where(order < int(0.57 * n), (u * low).long(), low + (u * (build - low)).long()).clamp_(max=build - 1)
        fk = torch.where(order < int(0.95 * n), dk[row], (build + u * (build // 20)).to(torch.int32))
        return {"fk": fk, "qty": _ints(g, n, 1, 100, torch.int32), "price": _doubles(g, n) * 100, "dk": dk, "cat": cat}
    assert kind == "pairs", kind
    build, keys = case["build"], case["keys"]
    rk = (torch.linspace(0, 1, build + 1, device=DEV, dtype=torch.float64)[:-1].pow(1.5) * keys).long()
    lk = torch.arange(n, device=DEV) % (keys + keys // 10)
    return {"lk": lk[torch.randperm(n, generator=g, device=DEV)], "a": _doubles(g, n),
            "rk": rk[torch.randperm(build, generator=g, device=DEV)], "b": _doubles(g, build)}


# ---- what a program holds before the query -----------------------------------------------------------------

_names = itertools.count()
_cache_ready = []
_streams = []


class _Table:
    """A cached table that leaves the cache with its last user."""

    def __init__(self, columns):
        if not _cache_ready:
            ColumnCache.init(0.5)
            _cache_ready.append(True)
        self.ref = GpuTableRef("memory", "perf", "t%d" % next(_names))
        torch.cuda.synchronize()
        ColumnCache.put_table(self.ref, columns)

    def __del__(self):
        try:
            ColumnCache.invalidate_table(self.ref)
        except Exception:
            pass


_TYPES = {torch.int16: T.INT16, torch.int32: T.INT32, torch.int64: T.INT64, torch.float32: T.FLOAT32,
          torch.float64: T.FLOAT64, torch.bool: T.BOOLEAN}


def _device(name, t):
    return make_device_column(name, _TYPES[t.dtype], t.data_ptr(), t.numel())


def _device_columns(cols, names):
    return [_device(n, cols[n]) for n in names]


def _stream():
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _cold_plan():
    scan = make_scan(["region", "open", "qty", "price"], GpuTableRef("memory", "perf", "cold"))
    filt = make_filter([make_expr("((bool*)out)[idx] = ((const bool*)inputs[0])[row];", ["open"], T.BOOLEAN)], scan)
    return make_group_by(["region"], [make_aggregate(A.SUM, "qty", T.HUGEINT), make_aggregate(A.AVG, "price", T.FLOAT64),
                                      make_aggregate(A.MAX, "qty", T.INT32), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         filt)


def _sum_plan(key):
    return make_group_by([key], [make_aggregate(A.SUM, "v", T.FLOAT64), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan([key, "v"], GpuTableRef("memory", "perf", "facts")))


def _star_plan():
    join = make_join("fk", "dk", ["qty", "price", "cat"], make_scan(["fk", "qty", "price"], GpuTableRef("memory", "perf", "fact")),
                     make_scan(["dk", "cat"], GpuTableRef("memory", "perf", "dim")))
    filt = make_filter([make_expr("((bool*)out)[idx] = (((const int*)inputs[0])[row] < 600);", ["cat"], T.BOOLEAN)], join)
    return make_projection([
        make_expr("((int*)out)[idx] = ((const int*)inputs[0])[row];", ["cat"], T.INT32),
        make_expr("((double*)out)[idx] = ((const double*)inputs[0])[row] * (double)((const int*)inputs[1])[row];",
                  ["price", "qty"], T.FLOAT64),
    ], filt)


def _pairs_plan():
    return make_join("lk", "rk", ["lk", "a", "b"], make_scan(["lk", "a"], GpuTableRef("memory", "perf", "left")),
                     make_scan(["rk", "b"], GpuTableRef("memory", "perf", "right")))


def _batch_plan(table, v_lt, w_mod):
    plan = c0_plan(v_lt, w_mod, table)
    plan.aggregates = plan.aggregates[:2]  # SUM and COUNT(*)
    return plan


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case, "inputs": [], "options": ExecuteOptions()}
    if kind == "batch":
        tables, plans = [], []
        for i, (rows, groups, v_lt, w_mod) in enumerate(_batch_shapes(case)):
            cols = _dash_inputs(_gen(seed, i + 1), rows, groups, v_lt, w_mod)
            tables.append(_Table(_device_columns(cols, ["k", "v", "w"])))
            plans.append(_batch_plan(tables[-1].ref, v_lt, w_mod))
        state.update(tables=tables, batch=GpuEngine.instance().prepare_batch(plans),
                     options=ExecuteOptions(serve_whole_scan_from_cache=True), inputs=[[] for _ in plans])
        return state
    cols = _inputs(case, seed)
    on_stream = _stream().cuda_stream
    if kind == "group":
        state["table"] = _Table(_device_columns(cols, ["k", "v", "w"]))
        state["plan"] = c0_plan(0.5, 7, state["table"].ref)
        state["options"] = ExecuteOptions(serve_whole_scan_from_cache=True)
    elif kind == "cold":
        host = {n: t.cpu().numpy() for n, t in cols.items()}
        state["plan"] = _cold_plan()
        state["inputs"] = [make_column("region", T.INT16, host["region"]), make_column("open", T.BOOLEAN, host["open"]),
                           make_column("qty", T.INT32, host["qty"]), make_column("price", T.FLOAT32, host["price"])]
    elif kind == "select":
        table = _device_columns(cols, ["k", "v", "w"])
        if case["nulls"]:  # a validity mask is staged from the host
            table[1] = make_column("v", T.FLOAT64, cols["v"].cpu().numpy(), cols["v_valid"].cpu().numpy())
        state["table"] = _Table(table)
        state["plan"] = cp_plan(0.5, 7, state["table"].ref)
        state["options"] = ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True, stream=on_stream)
    elif kind == "rollup" and case["skew"]:
        state["table"] = _Table(_device_columns(cols, ["a", "b", "amt", "v", "ts"]))
        state["plan"] = c1_plan(TS_MID, state["table"].ref)
        state["options"] = ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True, stream=on_stream)
    else:
        names = {"rollup": ["a", "v"], "ids": ["id", "v"], "join": ["pkey", "x", "bkey", "g"],
                 "star": ["fk", "qty", "price", "dk", "cat"], "pairs": ["lk", "a", "rk", "b"]}[kind]
        state["tensors"] = cols
        state["inputs"] = _device_columns(cols, names)
        state["plan"] = {"rollup": lambda: _sum_plan("a"), "ids": lambda: _sum_plan("id"), "join": c2_plan,
                         "star": _star_plan, "pairs": _pairs_plan}[kind]()
        state["options"] = ExecuteOptions(output_on_device=kind != "join", stream=on_stream)
    torch.cuda.synchronize()
    return state


# ---- one query ---------------------------------------------------------------------------------------------


class _View:
    """A device column of a result for torch: the tensor made from it keeps the result alive. The two words
    of a HUGEINT move as one 16-byte element."""

    _KINDS = {T.INT32: "<i4", T.INT64: "<i8", T.FLOAT64: "<f8", T.HUGEINT: "<c16"}

    def __init__(self, result, column):
        self.result = result
        self.__cuda_array_interface__ = {"shape": (column.row_count,), "typestr": self._KINDS[column.type],
                                         "data": (column.device_ptr, False), "version": 3, "strides": None}


def _tensors(result):
    return [torch.as_tensor(_View(result, c), device=DEV) for c in result.columns]


def _host(column):
    return column.data.view("<i8").reshape(-1, 2) if column.type == T.HUGEINT else column.data


def _checked(result):
    if getattr(result, "success", True) is not True:
        raise RuntimeError(result.error_message)
    return result


def _dense(index, columns, size):
    out = []
    for c in columns:
        table = torch.zeros(size, device=DEV, dtype=c.dtype)
        table[index] = c
        out.append(torch.view_as_real(table).view(torch.int64) if table.is_complex() else table)
    return out


def run(state):
    kind, engine = state["kind"], GpuEngine.instance()
    if kind == "batch":
        results, _ = engine.execute_batch(state["batch"], state["inputs"], state["options"])
        return [[_host(c) for c in _checked(r).columns] for r in results]
    result = _checked(engine.execute_plan(state["plan"], state["inputs"], state["options"]))
    if kind in ("group", "cold", "join"):
        return [_host(c) for c in result.columns]
    with torch.cuda.stream(_stream()):
        columns = _tensors(result)
        if kind == "rollup" and state["case"]["skew"]:
            index = columns[0].long() * ROLLUP_B + columns[1]
            return _dense(index, columns[2:], state["case"]["keys"] * ROLLUP_B)
        if kind == "rollup":
            return _dense(columns[0].long(), columns[1:], state["case"]["keys"])
        if kind == "ids":
            ids, order = torch.sort(columns[0])
            return [ids] + [c[order] for c in columns[1:]]
        return columns


# ---- the work of a query, and its result in 64 bits ------------------------------------------------------------


def work(case):
    kind, n = case["kind"], case.get("rows", 0)
    if kind == "group":
        return {"bytes": 20 * n + 36 * case["groups"], "flops": 2 * n}
    if kind == "cold":
        return {"bytes": 11 * n + 38 * case["groups"], "flops": n}
    if kind == "select":
        kept = 0.5 * (6 / 7) * (0.9 if case["nulls"] else 1.0)
        return {"bytes": int(n * (20 * (1 + kept) + (0.125 if case["nulls"] else 0))), "flops": 2 * n}
    if kind == "rollup" and case["skew"]:
        groups = min(case["keys"] * ROLLUP_B, n // 2)
        return {"bytes": int(32 * n + 0.35 * groups * 48), "flops": n}
    if kind == "rollup":
        return {"bytes": 12 * n + 20 * min(case["keys"], n), "flops": n}
    if kind == "ids":
        return {"bytes": 16 * n + 24 * min(case["keys"], n), "flops": n}
    if kind == "join":
        return {"bytes": 16 * n + 12 * case["build"], "flops": n}
    if kind == "star":
        return {"bytes": int(16 * n + 8 * case["build"] + 0.95 * 0.6 * 12 * n), "flops": n}
    if kind == "pairs":
        out = n / 1.1 * case["build"] / case["keys"]
        return {"bytes": int(16 * n + 16 * case["build"] + 24 * out), "flops": n}
    rows = sum(s[0] for s in _batch_shapes(case))
    return {"bytes": 20 * rows, "flops": 2 * rows}


def _sums(index, values, size):
    return torch.zeros(size, device=DEV, dtype=torch.float64).index_add_(0, index, values.double())


def _dash_exact(cols, groups, v_lt, w_mod):
    keep = (cols["v"] < v_lt) & (cols["w"] % w_mod != 0)
    k, v = cols["k"][keep].long(), cols["v"][keep]
    return _sums(k, v * 2.0 + 1.0, groups)[torch.bincount(k, minlength=groups) > 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [[None, _dash_exact(_dash_inputs(_gen(seed, i + 1), rows, groups, v_lt, w_mod), groups, v_lt, w_mod),
                 None]
                for i, (rows, groups, v_lt, w_mod) in enumerate(_batch_shapes(case))]
    cols = _inputs(case, seed)
    if kind == "group":
        return [None, _dash_exact(cols, case["groups"], 0.5, 7), None, None, None]
    if kind == "cold":
        k = cols["region"][cols["open"]].long() + 5
        count = torch.bincount(k, minlength=case["groups"])
        mean = _sums(k, cols["price"][cols["open"]], case["groups"]) / count
        return [None, None, mean[count > 0], None, None]
    if kind == "select":
        keep = (cols["v"] < 0.5) & (cols["w"] % 7 != 0)
        if case["nulls"]:
            keep &= cols["v_valid"]
        return [None, cols["v"][keep] * 2.0 + 1.0, None]
    if kind == "rollup" and case["skew"]:
        keep = cols["ts"] > TS_MID
        k = cols["a"][keep].long() * ROLLUP_B + cols["b"][keep]
        size = case["keys"] * ROLLUP_B
        count = torch.bincount(k, minlength=size)
        return [None, _sums(k, cols["v"][keep], size) / count.clamp(min=1), None, None]
    if kind == "rollup":
        return [_sums(cols["a"].long(), cols["v"], case["keys"]), None]
    if kind == "ids":
        _, k = torch.unique(cols["id"], return_inverse=True)
        return [None, _sums(k, cols["v"], int(k.max()) + 1), None]
    if kind == "join":
        hit = cols["pkey"] < case["build"]
        table = torch.empty(case["build"], device=DEV, dtype=torch.int64)
        table[cols["bkey"]] = cols["g"].long()
        return [None, _sums(table[cols["pkey"][hit]], cols["x"][hit], min(case["build"], JOIN_GROUPS))]
    if kind == "star":
        table = torch.full((case["build"] + case["build"] // 20 + 1,), 1000, device=DEV, dtype=torch.int64)
        table[cols["dk"].long()] = cols["cat"].long()
        keep = table[cols["fk"].long()] < 600  # 1000: not in the dimension
        return [None, (cols["price"] * cols["qty"].double())[keep]]
    rk, order = torch.sort(cols["rk"], stable=True)
    first = torch.searchsorted(rk, cols["lk"], right=False)
    count = torch.searchsorted(rk, cols["lk"], right=True) - first
    left = torch.repeat_interleave(count)
    start = torch.cumsum(count, 0) - count
    within = torch.arange(left.numel(), device=DEV) - start[left]
    return [None, cols["a"][left], cols["b"][order[first[left] + within]]]
