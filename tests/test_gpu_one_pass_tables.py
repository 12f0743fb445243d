"""The one-pass group-by's shared-memory tables on the B200 against numpy: key spaces from one slot (thirty-two
copies of it) to the largest, sums of doubles that stand for a group's presence -- negative zeros, infinities,
NaN and sums that cancel --, rows around the launch shapes' bounds, and joins whose probe reads two rows a thread."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column, make_expr,
                           make_filter, make_group_by, make_join, make_scan)
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, hugeint_to_int

pytestmark = pytest.mark.gpu


def _run(plan, inputs, options=None):
    r = GpuEngine.instance().execute_plan(plan, inputs, options)
    assert r.success, r.error_message
    return r.columns


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("rows", [1, 2047, 2049, 70_001, 700_001])
@pytest.mark.parametrize("groups", [1, 2, 3, 31, 64, 129, 500, 1023])
def test_every_state_over_every_number_of_copies(groups, rows, cached):
    rng = np.random.default_rng(groups * 7 + rows)
    k = rng.integers(0, groups, rows).astype(np.int32) + 40
    k[0], k[-1] = 40, 40 + groups - 1
    v = rng.integers(-(1 << 62), 1 << 62, rows, dtype=np.int64)
    w = rng.integers(-(1 << 31) + 9, (1 << 31) - 9, rows).astype(np.int64)
    x = rng.integers(-1000, 1000, rows).astype(np.float64)
    cols = [make_column("k", T.INT32, k), make_column("v", T.INT64, v), make_column("w", T.INT64, w), make_column("x", T.FLOAT64, x)]
    ref = GpuTableRef("memory", "main", "copies")
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT), make_aggregate(A.MIN, "w", T.INT64),
                                 make_aggregate(A.MAX, "v", T.INT64), make_aggregate(A.SUM, "x", T.FLOAT64),
                                 make_aggregate(A.COUNT_STAR, "", T.INT64)], make_scan(["k", "v", "w", "x"], ref))
    if cached:
        ColumnCache.put_table(ref, cols)
        try:
            got = _run(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True))
        finally:
            ColumnCache.invalidate_table(ref)
    else:
        got = _run(plan, cols)
    keys, inv = np.unique(k, return_inverse=True)
    sums = [0] * len(keys)
    for i, a in zip(inv.tolist(), v.tolist()):
        sums[i] += a
    lo, hi = np.full(len(keys), np.iinfo(np.int64).max), np.full(len(keys), np.iinfo(np.int64).min)
    np.minimum.at(lo, inv, w)
    np.maximum.at(hi, inv, v)
    assert np.array_equal(got[0].data, keys) and hugeint_to_int(got[1].data) == sums
    assert np.array_equal(got[2].data, lo) and np.array_equal(got[3].data, hi)
    assert np.array_equal(got[4].data, np.bincount(inv, weights=x)) and np.array_equal(got[5].data, np.bincount(inv))


@pytest.mark.parametrize("groups", [7, 900, 4096])
def test_double_sums_that_mark_their_groups(groups):
    """Only sums of doubles: a group exists exactly when it has rows, whatever they add up to."""
    rng = np.random.default_rng(groups)
    n = 300_007
    k = rng.integers(0, groups, n).astype(np.int32)
    k[k == 2] = 3  # no rows
    x = rng.integers(-1000, 1000, n).astype(np.float64)
    x[k == 0] = -0.0  # sums to zero
    x[k == 1] = np.where(np.arange((k == 1).sum()) % 2 == 0, 5.0, -5.0)  # cancels, or leaves one 5
    x[np.flatnonzero(k == 4)[:1]] = np.inf
    x[np.flatnonzero(k == 5)[:1]] = np.nan
    x[np.flatnonzero(k == 6)[:2]] = [np.inf, -np.inf]
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "x", T.FLOAT64), make_aggregate(A.SUM, "y", T.FLOAT64)],
                         make_scan(["k", "x", "y"]))
    got = _run(plan, [make_column("k", T.INT32, k), make_column("x", T.FLOAT64, x),
                      make_column("y", T.FLOAT32, np.full(n, 0.5, np.float32))])
    keys, inv = np.unique(k, return_inverse=True)
    with np.errstate(invalid="ignore"):
        want = np.bincount(inv, weights=x)
    assert np.array_equal(got[0].data, keys)
    assert np.array_equal(got[1].data, want, equal_nan=True)
    assert not np.signbit(got[1].data[0]) and got[1].data[0] == 0.0
    assert np.array_equal(got[2].data, np.bincount(inv) * 0.5)


def test_double_sums_over_a_filter_that_keeps_nothing():
    k = np.arange(5000, dtype=np.int32) % 50
    filt = make_filter([make_expr("((bool*)out)[idx] = ((const double*)inputs[0])[row] > 9.0;", ["x"], T.BOOLEAN)], make_scan(["k", "x"]))
    got = _run(make_group_by(["k"], [make_aggregate(A.SUM, "x", T.FLOAT64)], filt),
               [make_column("k", T.INT32, k), make_column("x", T.FLOAT64, np.ones(5000))])
    assert [len(c.data) for c in got] == [0, 0]


@pytest.mark.parametrize("kt,vt,rows", [(T.INT16, T.INT16, 10_001), (T.INT16, T.BOOLEAN, 2_047), (T.INT32, T.INT64, 65_537),
                                        (T.INT64, T.FLOAT64, 500_001)])
def test_join_probe_of_narrow_and_wide_columns(kt, vt, rows):
    """Two rows of a 1- or 2-byte column are read as they come, wider ones in one access."""
    np_t = {T.INT16: np.int16, T.BOOLEAN: np.uint8, T.INT32: np.int32, T.INT64: np.int64, T.FLOAT64: np.float64}
    rng = np.random.default_rng(rows)
    rk = rng.permutation(3000).astype(np_t[kt])
    rg = rng.integers(0, 700, 3000).astype(np.int32)
    lk = rng.integers(0, 3300, rows).astype(np_t[kt])
    lv = rng.integers(0, 2, rows).astype(np_t[vt])
    agg = make_aggregate(A.MAX, "lv", vt) if vt == T.BOOLEAN else make_aggregate(A.SUM, "lv", T.FLOAT64 if vt == T.FLOAT64 else T.HUGEINT)
    plan = make_group_by(["rg"], [agg], make_join("lk", "rk", ["rg", "lv"], make_scan(["lk", "lv"]), make_scan(["rk", "rg"])))
    got = _run(plan, [make_column("lk", kt, lk), make_column("lv", vt, lv), make_column("rk", kt, rk), make_column("rg", T.INT32, rg)])
    g = np.full(3300, -1)
    g[rk] = rg
    hit = g[lk] >= 0
    keys, inv = np.unique(g[lk[hit]], return_inverse=True)
    assert np.array_equal(got[0].data, keys)
    if vt == T.BOOLEAN:
        best = np.zeros(len(keys), np.uint8)
        np.maximum.at(best, inv, lv[hit])
        assert np.array_equal(got[1].data, best)
    else:
        want = np.bincount(inv, weights=lv[hit].astype(np.float64))
        have = got[1].data if vt == T.FLOAT64 else np.array(hugeint_to_int(got[1].data), np.float64)
        assert np.array_equal(have, want)
