"""Memory of the one-pass row filter on the B200: a result on the device holds little more than its rows, whole columns
of one result stay readable while it lives, and a filter below another operator leaves a tight budget to that one."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, device_to_host, make_column, make_expr,
                           make_filter, make_join, make_scan)
from vectisdb_b200.abi import check, lib
from vectisdb_b200.engine import GpuValueType as T, memory_reset_peak, memory_stats, profile_drain, profile_enable

pytestmark = pytest.mark.gpu


def _below(bound, scan):
    return make_filter([make_expr(f"((bool*)out)[idx] = (((const int*)inputs[0])[row] < {bound});", ["x"], T.BOOLEAN)], scan)


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("rows,keep", [(100_003, 1), (1_000_003, 0), (1_000_003, 1), (1_000_003, 24), (3_000_017, 1)])
def test_few_rows_kept_hold_little(rows, keep, nulls):
    x = (np.arange(rows) % 100).astype(np.int32)
    d = np.arange(rows, dtype=np.float64)
    valid = np.arange(rows) % 7 != 0
    ref = GpuTableRef("memory", "main", "room")
    ColumnCache.put_table(ref, [make_column("x", T.INT32, x), make_column("d", T.FLOAT64, d, valid if nulls else None)])
    try:
        before = memory_stats()["in_use_bytes"]
        r = GpuEngine.instance().execute_plan(_below(keep, make_scan(["x", "d"], ref)), [],
                                              ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True))
        held = memory_stats()["in_use_bytes"] - before
        got = [device_to_host(c) for c in r.columns]
        r.free()
        assert held <= (x < keep).sum() * 14 + (4 << 20) + 4096, held
        assert np.array_equal(got[0], x[x < keep])
        sure = valid[x < keep] if nulls else slice(None)
        assert np.array_equal(got[1][sure], d[x < keep][sure])
        assert memory_stats()["in_use_bytes"] == before
    finally:
        ColumnCache.invalidate_table(ref)


def test_a_filter_below_a_join_leaves_the_budget_to_it(monkeypatch):
    rng = np.random.default_rng(2)
    n = 4_000_003
    x = (np.arange(n) % 3).astype(np.int32)
    rk = rng.permutation(n).astype(np.int64)
    lk = rng.integers(0, n, 5000).astype(np.int64)
    refs = [GpuTableRef("memory", "main", "room_" + s) for s in ("left", "right")]
    ColumnCache.put_table(refs[0], [make_column("lk", T.INT64, lk)])
    ColumnCache.put_table(refs[1], [make_column("x", T.INT32, x), make_column("rk", T.INT64, rk)])
    plan = make_join("lk", "rk", ["lk", "x"], make_scan(["lk"], refs[0]), _below(1, make_scan(["x", "rk"], refs[1])))

    def run():
        profile_drain()
        profile_enable(True)
        memory_reset_peak()
        before = memory_stats()["in_use_bytes"]
        try:
            r = GpuEngine.instance().execute_plan(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True))
            names = [rec[0] for rec in profile_drain()]
        finally:
            profile_enable(False)
        return r, names, memory_stats()["peak_bytes"] - before
    try:
        r, names, wide = run()
        assert r.success and "vgpu_mat_onepass" in names, names
        monkeypatch.setenv("VGPU_MAT_PASSES", "2")
        r, names, narrow = run()
        monkeypatch.delenv("VGPU_MAT_PASSES")
        assert r.success and narrow < wide, (narrow, wide)
        check(lib().vgpu_memory_set_budget(memory_stats()["in_use_bytes"] + narrow))
        try:
            r, _, _ = run()
        finally:
            check(lib().vgpu_memory_set_budget(0))
        assert r.success, r.error_message
        kept = set(rk[x < 1].tolist())
        assert np.array_equal(r.columns[0].data, [k for k in lk.tolist() if k in kept])
    finally:
        for ref in refs:
            ColumnCache.invalidate_table(ref)
