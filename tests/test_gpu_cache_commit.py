"""Committing staged columns on the B200 when memory runs out on the way: the columns that were finished are cached with
their ranges, and nothing is lost to the allocator."""
import numpy as np
import pytest

from vectisdb_b200 import ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column, make_group_by, make_scan
from vectisdb_b200.abi import VgpuError, check, lib
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, memory_stats

pytestmark = pytest.mark.gpu


def test_finished_columns_are_kept_when_a_later_one_fails():
    n = 1 << 20
    a = (np.arange(2 * n) % 700 - 300).astype(np.int16)
    ref = GpuTableRef("memory", "main", "commit")
    ColumnCache.init(0.5)
    before = memory_stats()["in_use_bytes"]
    ColumnCache.begin_staging(ref)
    for half in (slice(0, n), slice(n, 2 * n)):
        assert ColumnCache.stage_chunk(ref, make_column("b", T.INT64, np.arange(n)))
        assert ColumnCache.stage_chunk(ref, make_column("a", T.INT16, a[half]))
    try:
        # room to join the halves of "a" (4 bytes a row of the half), not those of "b" (16)
        check(lib().vgpu_memory_set_budget(memory_stats()["in_use_bytes"] + 8 * n))
        try:
            with pytest.raises(VgpuError, match="budget"):
                ColumnCache.commit_staging(ref, 2 * n)
        finally:
            check(lib().vgpu_memory_set_budget(0))
        plan = make_group_by(["a"], [make_aggregate(A.COUNT_STAR, "", T.INT64)], make_scan(["a"], ref))
        r = GpuEngine.instance().execute_plan(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True))
        assert r.success, r.error_message
        keys, counts = np.unique(a, return_counts=True)
        assert np.array_equal(r.columns[0].data, keys) and np.array_equal(r.columns[1].data, counts)
        ColumnCache.commit_staging(ref, 2 * n)  # the other one, now that there is room
        assert ColumnCache.replayable_chunk_rows(ref, ["a", "b"]) == [n, n]
    finally:
        ColumnCache.abort_staging(ref)
        ColumnCache.invalidate_table(ref)
    assert memory_stats()["in_use_bytes"] == before
