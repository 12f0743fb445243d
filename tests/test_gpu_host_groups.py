"""Groups written straight to page-locked host memory by the one-pass group-by on the B200: results on either
side of the size bound, many results alive at once, several threads, no groups, and a group-by below the root
(whose rows stay on the device)."""
import threading

import numpy as np
import pytest

from vectisdb_b200 import (GpuEngine, make_aggregate, make_column, make_expr, make_filter, make_group_by, make_scan)
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, hugeint_to_int

pytestmark = pytest.mark.gpu


def _query(seed, n, groups, aggs=1):
    rng = np.random.default_rng(seed)
    k = rng.integers(-3, groups - 3, n).astype(np.int16)
    v = rng.integers(-(1 << 40), 1 << 40, n).astype(np.int64)
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT)] * aggs + [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["k", "v"]))
    keys, inv = np.unique(k, return_inverse=True)
    sums = [0] * len(keys)
    for i, x in zip(inv.tolist(), v.tolist()):
        sums[i] += x
    return plan, [make_column("k", T.INT16, k), make_column("v", T.INT64, v)], (keys, sums, np.bincount(inv))


def _check(result, expected, aggs=1):
    assert result.success, result.error_message
    keys, sums, counts = expected
    assert np.array_equal(result.columns[0].data, keys)
    for i in range(aggs):
        assert hugeint_to_int(result.columns[1 + i].data) == sums
    assert np.array_equal(result.columns[-1].data, counts)


@pytest.mark.parametrize("groups,aggs", [(1, 1), (2, 1), (1000, 1), (1024, 5), (4096, 1), (1024, 15)])
def test_sizes_on_either_side_of_the_bound(groups, aggs):
    """1024 slots with fifteen sums take 0.25 MB and some: copied as before."""
    plan, cols, expected = _query(groups + aggs, 30_001, groups, aggs)
    _check(GpuEngine.instance().execute_plan(plan, cols), expected, aggs)


def test_many_results_alive_at_once():
    queries = [_query(s, 5000 + s, 50 + 3 * s) for s in range(40)]
    results = [GpuEngine.instance().execute_plan(plan, cols) for plan, cols, _ in queries]
    for r, (_, _, expected) in zip(results, queries):
        _check(r, expected)


def test_several_threads():
    failures = []

    def work(seed):
        try:
            for i in range(15):
                plan, cols, expected = _query(seed * 100 + i, 3000, 40)
                _check(GpuEngine.instance().execute_plan(plan, cols), expected)
        except BaseException as e:  # noqa: BLE001 -- reported by the main thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_no_groups_and_a_group_by_below_the_root():
    plan, cols, (keys, sums, counts) = _query(5, 20_000, 300)
    none = make_filter([make_expr("((bool*)out)[idx] = ((const short*)inputs[0])[row] > 10000;", ["k"], T.BOOLEAN)],
                       plan.children[0])
    r = GpuEngine.instance().execute_plan(make_group_by(["k"], plan.aggregates, none), cols)
    assert r.success and [len(c.data) for c in r.columns] == [0, 0, 0]
    above = make_group_by(["agg_1"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                          make_group_by(["k"], [make_aggregate(A.MAX, "v", T.INT64), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                                        plan.children[0]))
    r = GpuEngine.instance().execute_plan(above, cols)
    values, times = np.unique(counts, return_counts=True)
    assert r.success and np.array_equal(r.columns[0].data, values) and np.array_equal(r.columns[1].data, times)
