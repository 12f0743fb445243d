"""Host results of a batch on the B200: each query's columns are in memory of its own, so that a column which is kept
holds its query's buffer alone and the others' serve the next call."""
import gc

import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, GpuTableRef, make_column
from vectisdb_b200 import workloads as W
from vectisdb_b200.engine import GpuValueType as T

pytestmark = pytest.mark.gpu


def _query(rng, rows, groups):
    k = rng.integers(0, groups, rows).astype(np.int32)
    k[:2] = [0, groups - 1]
    return [make_column("k", T.INT32, k), make_column("v", T.FLOAT64, rng.random(rows) * 0.4),
            make_column("w", T.INT64, rng.integers(1, 7, rows, dtype=np.int64))]


def _keys(columns):
    return np.unique(columns[0].data)


def test_a_kept_column_holds_its_own_query_alone():
    rng = np.random.default_rng(3)
    queries = [_query(rng, 300_000, 1 << 17), _query(rng, 5000, 50), _query(rng, 90_000, 3000), _query(rng, 400, 7)]
    plans = [W.c0_plan(0.5, 7, GpuTableRef("memory", "main", f"bm{i}")) for i in range(len(queries))]

    def run():
        results, stats = GpuEngine.instance().execute_batch(plans, queries)
        assert stats["batched"] == len(queries), stats
        for q, r in zip(queries, results):
            assert np.array_equal(r.columns[0].data, _keys(q))
        return results
    first = run()
    kept = first[1].columns[0].data  # of a small query
    large = first[0].columns[0].data.ctypes.data
    del first
    gc.collect()
    for _ in range(3):
        again = run()
        assert again[0].columns[0].data.ctypes.data == large  # the large query's buffer came back
        assert np.array_equal(kept, _keys(queries[1]))
        del again
        gc.collect()
