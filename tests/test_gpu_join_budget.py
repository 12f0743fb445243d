"""The materializing join's grouped right rows against the device-memory budget on the B200: where their entries do not
fit, or the outputs beside them do not, the right keys are sorted, as long as that fits."""
import numpy as np
import pytest

from vectisdb_b200 import ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_column, make_join, make_scan
from vectisdb_b200.abi import check, lib
from vectisdb_b200.engine import GpuValueType as T, memory_reset_peak, memory_stats, profile_drain, profile_enable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left,extra", [(1000, 1 << 20), (1000, 6 << 20), (50_000, 4 << 20)])
def test_the_sort_runs_where_the_entries_do_not_fit(left, extra):
    rng = np.random.default_rng(left)
    n = 1_000_003
    rk = rng.permutation(n).astype(np.int64) * 4  # 8 bytes for each of four key values a row
    rk[0], rk[1] = rk[1], rk[1]  # one key twice
    lk = rng.integers(0, 4 * n, left).astype(np.int64)
    b = rng.standard_normal(n)
    refs = [GpuTableRef("memory", "main", "jb_" + s) for s in ("left", "right")]
    ColumnCache.put_table(refs[0], [make_column("lk", T.INT64, lk)])
    ColumnCache.put_table(refs[1], [make_column("rk", T.INT64, rk), make_column("b", T.FLOAT64, b)])
    plan = make_join("lk", "rk", ["lk", "b"], make_scan(["lk"], refs[0]), make_scan(["rk", "b"], refs[1]))

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
        assert r.success and "radix_scatter" not in names, names
        # the sort: keys and positions twice over, then keys, positions, a directory and the left rows' ranges
        room = max(24 * n, 28 * n + 24 * left + r.columns[0].row_count * 24) + extra
        check(lib().vgpu_memory_set_budget(memory_stats()["in_use_bytes"] + min(room, wide - (1 << 20))))
        try:
            r, names, _ = run()
        finally:
            check(lib().vgpu_memory_set_budget(0))
        assert r.success, r.error_message
        assert "radix_scatter" in names, names
    finally:
        for ref in refs:
            ColumnCache.invalidate_table(ref)
    order = np.argsort(rk, kind="stable")
    first = np.searchsorted(rk[order], lk, side="left")
    count = np.searchsorted(rk[order], lk, side="right") - first
    at = np.repeat(np.arange(left), count)
    right = order[first[at] + np.arange(len(at)) - np.repeat(np.cumsum(count) - count, count)]
    assert np.array_equal(r.columns[0].data, lk[at]) and np.array_equal(r.columns[1].data, b[right])
