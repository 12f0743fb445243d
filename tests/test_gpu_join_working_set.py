"""The working-set estimate of a join under a group-by against what it allocates, right keys cached: ranges of nearly
four values a row, values of every table width, and dense keys that repeat, which are sorted in the end."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column,
                           make_group_by, make_join, make_scan)
from vectisdb_b200.engine import (GpuAggregateKind as A, GpuValueType as T, estimate_working_set_for,
                                  memory_reset_peak, memory_stats)

pytestmark = pytest.mark.gpu
ROWS = 1 << 20


@pytest.mark.parametrize("keys,values", [("spread", "wide"), ("spread", "float"), ("spread", "two"), ("dense", "float"),
                                         ("repeated", "two"), ("repeated", "long")])
def test_estimate_against_allocations(keys, values, monkeypatch):
    monkeypatch.setenv("VGPU_JOIN_CACHE", "0")  # every run builds its table
    rng = np.random.default_rng(5)
    rk = rng.permutation(ROWS).astype(np.int32)
    if keys == "spread":
        rk = rk * 4 - (rk > 0)  # range 4 * rows - 5
    elif keys == "repeated":
        rk = rk // 300
    g = (np.arange(ROWS) % 1000).astype(np.int32)
    right = [make_column("rk", T.INT32, rk), make_column("g", T.INT32, g)]
    if values == "wide":  # offsets past 16 bits
        right[1] = make_column("g", T.INT32, np.where(g == 0, 1 << 17, g).astype(np.int32))
    extra = {"float": T.FLOAT32, "two": T.INT32, "long": T.INT64}.get(values)
    if extra:
        right.append(make_column("y", extra, np.arange(ROWS)))
    left = [make_column("lk", T.INT32, rk[:4096])]
    refs = [GpuTableRef("memory", "main", "ws_" + s) for s in ("left", "right")]
    ColumnCache.put_table(refs[0], left)
    ColumnCache.put_table(refs[1], right)
    key, outs, aggs = (["lk"], ["lk", "y"], [make_aggregate(A.SUM, "y", T.FLOAT64)]) if values == "float" else \
        (["g"], ["g"] + (["y"] if extra else []), [make_aggregate(A.COUNT_STAR, "", T.INT64)] +
         ([make_aggregate(A.MAX, "y", extra)] if extra else []))
    plan = make_group_by(key, aggs, make_join("lk", "rk", outs, make_scan(["lk"], refs[0]),
                                              make_scan([c.name for c in right], refs[1])))
    options = ExecuteOptions(serve_whole_scan_from_cache=True)
    try:
        predicted = estimate_working_set_for(plan, [], options).total_bytes
        memory_reset_peak()
        before = memory_stats()["in_use_bytes"]
        r = GpuEngine.instance().execute_plan(plan, [], options)
        measured = memory_stats()["peak_bytes"] - before
    finally:
        for ref in refs:
            ColumnCache.invalidate_table(ref)
    assert r.success, r.error_message
    assert 0.4 <= predicted / measured <= 4.0, (predicted, measured)  # the band of the working-set estimate
