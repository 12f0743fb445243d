"""Batched group-by over tables of one and of several segments, on the B200, against numpy: key spaces at the edges
of a segment, segments without groups, row counts at the edges of a tile, filters that keep nothing, and repeated runs
over accumulators that the run before has to leave clean."""
import numpy as np
import pytest

from vectisdb_b200 import BatchOptions, GpuEngine, GpuTableRef, make_column
from vectisdb_b200 import workloads as W
from vectisdb_b200.engine import GpuValueType as T

pytestmark = pytest.mark.gpu


def _query(rng, rows, span, groups, v_lt):
    used = np.unique(np.concatenate([[0, span - 1], rng.integers(0, span, groups)]))
    k = rng.choice(used, rows).astype(np.int32) - 77
    k[0], k[-1] = -77, span - 78
    v, w = rng.random(rows), rng.integers(0, 1000, rows, dtype=np.int64)
    return [make_column("k", T.INT32, k), make_column("v", T.FLOAT64, v), make_column("w", T.INT64, w)], (k, v, w, v_lt)


def _check(columns, k, v, w, v_lt):
    keep = (v < v_lt) & (w % 7 != 0)
    uk, inv = np.unique(k[keep], return_inverse=True)
    got = [c.data for c in columns]
    assert np.array_equal(got[0], uk)  # in key order
    exp = np.bincount(inv, weights=v[keep] * 2.0 + 1.0, minlength=len(uk))  # the plan projects v * 2 + 1
    assert np.all(np.abs(got[1] - exp) <= 1e-12 * np.abs(exp))  # at most some 10^5 positive addends
    assert np.array_equal(got[2], np.bincount(inv, minlength=len(uk)))


@pytest.mark.parametrize("spans", [[2, 1023, 1024], [1025], [1024, 1025, 1 << 16, 3, 70_000], [(1 << 22) - 5, 2048, 2049]])
@pytest.mark.parametrize("tile_rows", [0, 1024])
def test_tables_of_one_and_of_several_segments(spans, tile_rows):
    rng = np.random.default_rng(8)
    sizes = [2, 1023, 4096, 4097, 100_003]
    queries = [_query(rng, sizes[(i + j) % len(sizes)], span, 300, v_lt)
               for i, span in enumerate(spans) for j, v_lt in enumerate([0.6, 0.0, 0.9, 0.5])]
    plans = [W.c0_plan(q[1][3], 7, GpuTableRef("memory", "main", f"seg{i}")) for i, q in enumerate(queries)]
    for _ in range(3):
        results, stats = GpuEngine.instance().execute_batch(plans, [q[0] for q in queries], batch=BatchOptions(tile_rows=tile_rows))
        assert stats["batched"] == len(queries), stats
        for q, r in zip(queries, results):
            _check(r.columns, *q[1])
