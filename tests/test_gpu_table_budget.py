"""Group-by tables in L2 against the device-memory budget and what a request was admitted for, on the B200: few rows
whose keys span millions of values, and sparse keys. What fits the partitioned form runs in it."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, Server, make_aggregate, make_column,
                           make_group_by, make_scan)
from vectisdb_b200.abi import check, lib
from vectisdb_b200.engine import (GpuAggregateKind as A, GpuValueType as T, memory_reset_peak, memory_stats,
                                  profile_drain, profile_enable)

pytestmark = pytest.mark.gpu
CACHED = ExecuteOptions(serve_whole_scan_from_cache=True)


def _case(kind):
    rng = np.random.default_rng(8)
    if kind == "dense":  # a slot of 16 bytes for each of 2^22 values: 64 MB
        k = rng.integers(0, 1 << 22, 4096)
        k[:2] = [0, (1 << 22) - 1]
    else:
        k = rng.integers(0, 1 << 50, 4096)
    x = rng.integers(0, 1000, len(k)).astype(np.float64)
    cols = [make_column("k", T.INT64, k), make_column("x", T.FLOAT64, x)]
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "x", T.FLOAT64), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["k", "x"], GpuTableRef("memory", "main", "budget_" + kind)))
    return plan, cols


def _check(columns, cols):
    keys, inv = np.unique(cols[0].data, return_inverse=True)
    order = np.argsort(columns[0].data)
    assert np.array_equal(columns[0].data[order], keys)
    assert np.array_equal(columns[1].data[order], np.bincount(inv, weights=cols[1].data))
    assert np.array_equal(columns[2].data[order], np.bincount(inv))


def _run(plan):
    profile_drain()
    profile_enable(True)
    memory_reset_peak()
    before = memory_stats()["in_use_bytes"]
    try:
        r = GpuEngine.instance().execute_plan(plan, [], CACHED)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    return r, names, memory_stats()["peak_bytes"] - before


@pytest.mark.parametrize("kind", ["dense", "sparse"])
def test_a_tight_budget_keeps_the_partitioned_form(kind, monkeypatch):
    plan, cols = _case(kind)
    table = plan.children[0].table
    ColumnCache.put_table(table, cols)
    try:
        r, names, wide = _run(plan)
        assert r.success and "vgpu_gb_l2" in names, names
        monkeypatch.setenv("VGPU_GB_STRATEGY", "hash")
        r, names, narrow = _run(plan)
        monkeypatch.delenv("VGPU_GB_STRATEGY")
        assert r.success and "vgpu_gb_l2" not in names and narrow < wide, (names, narrow, wide)
        check(lib().vgpu_memory_set_budget(memory_stats()["in_use_bytes"] + (narrow + wide) // 2))
        try:
            r, names, _ = _run(plan)
        finally:
            check(lib().vgpu_memory_set_budget(0))
        assert r.success, r.error_message
        assert "vgpu_gb_l2" not in names, names
        _check(r.columns, cols)
    finally:
        ColumnCache.invalidate_table(table)


@pytest.mark.parametrize("batch_max", [1, 8])
def test_a_served_request_stays_within_its_estimate(batch_max):
    plan, cols = _case("dense")
    server = Server(slots=2, batch_max=batch_max)
    try:
        server.wait(server.submit(plan, cols))  # compiled
        memory_reset_peak()
        before = memory_stats()["in_use_bytes"]
        result, info = server.wait(server.submit(plan, cols))
        peak = memory_stats()["peak_bytes"] - before
    finally:
        server.close()
    assert info["status"] == 0, info["error"]
    _check(result.columns, cols)
    assert peak <= info["estimated_bytes"] / 0.4, (peak, info)  # the band of the working-set estimate
