"""The launch count of a replayed batch on the B200: the graph's kernels, with the count of a table's segments where there
are several."""
import numpy as np
import pytest

from vectisdb_b200 import ExecuteOptions, ColumnCache, GpuEngine, GpuTableRef, make_column
from vectisdb_b200 import workloads as W
from vectisdb_b200.engine import GpuValueType as T, launch_count

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,launches", [(100, 2), (5000, 3)])
def test_launches_of_a_replayed_batch(groups, launches):
    import torch
    refs, plans = [], []
    for i in range(3):
        k = (np.arange(20_000) % groups).astype(np.int32)
        refs.append(GpuTableRef("memory", "main", f"bl{i}"))
        ColumnCache.put_table(refs[-1], [make_column("k", T.INT32, k), make_column("v", T.FLOAT64, np.full(20_000, 0.25)),
                                         make_column("w", T.INT64, np.ones(20_000, np.int64))])
        plans.append(W.c0_plan(0.5, 7, refs[-1]))
    options = ExecuteOptions(serve_whole_scan_from_cache=True, stream=torch.cuda.Stream().cuda_stream)
    try:
        batch = GpuEngine.instance().prepare_batch(plans)
        for _ in range(2):  # compiled, captured
            GpuEngine.instance().execute_batch(batch, [[]] * 3, options)
        before = launch_count()
        results, _ = GpuEngine.instance().execute_batch(batch, [[]] * 3, options)
        assert launch_count() - before == launches
        assert all(len(r.columns[0].data) == groups for r in results)
    finally:
        for ref in refs:
            ColumnCache.invalidate_table(ref)
