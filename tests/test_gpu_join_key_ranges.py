"""Group keys from a join's right side on the B200, grouped over the rows that the join keeps: right rows without a match
may hold any value, and do not count toward the bits that the keys are packed into."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_aggregate, make_column, make_group_by, make_join, make_scan
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, profile_drain, profile_enable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("repeat", [1, 2])
@pytest.mark.parametrize("keys", [("x", "y"), ("x", "y", "w"), ("x", "l"), ("g", "l")])
def test_unmatched_right_rows_do_not_widen_the_keys(keys, repeat):
    rng = np.random.default_rng(repeat)
    n = 5000
    rk = np.repeat(rng.permutation(n).astype(np.int64), repeat)
    met = rk < 3000
    wild = lambda bits: rng.integers(-(1 << bits), 1 << bits, len(rk))
    right = {"rk": (T.INT64, rk), "x": (T.INT64, np.where(met, wild(3), wild(61))), "y": (T.INT64, np.where(met, wild(4), wild(61))),
             "w": (T.INT32, np.where(met, wild(2), wild(30))), "g": (T.INT32, np.where(met, np.abs(wild(3)), np.abs(wild(30))))}
    lk = rng.integers(0, 3000, 20_001).astype(np.int64)  # every left row has matches
    left = {"lk": (T.INT64, lk), "l": (T.INT64, rng.integers(0, 1 << (34 if keys[0] == "g" else 40), len(lk)) // (1 << 31) * (1 << 31))}
    used = [k for k in keys if k in right]
    cols = [make_column(c, t, v) for c, (t, v) in list(left.items())] + [make_column(c, *right[c]) for c in ["rk"] + used]
    plan = make_group_by(list(keys), [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_join("lk", "rk", list(keys), make_scan(["lk", "l"]), make_scan(["rk"] + used)))
    r = GpuEngine.instance().execute_plan(plan, cols)
    assert r.success, r.error_message
    order = np.argsort(rk, kind="stable")
    first = np.searchsorted(rk[order], lk)
    at = (first[:, None] + np.arange(repeat)).ravel()
    rows = np.repeat(np.arange(len(lk)), repeat)
    packed = np.stack([np.asarray(left["l"][1][rows] if k == "l" else right[k][1][order[at]]).astype(np.int64) for k in keys], axis=1)
    groups, counts = np.unique(packed, axis=0, return_counts=True)
    got = np.stack([c.data.astype(np.int64) for c in r.columns[:-1]], axis=1)
    sort = np.lexsort(got.T[::-1])
    assert np.array_equal(got[sort], groups) and np.array_equal(r.columns[-1].data[sort], counts)


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("outlier", [False, True])
def test_an_unmatched_outlier_keeps_the_shared_memory_table(outlier, extra):
    """Two hundred codes and one far off that no left row meets; with a second right column they are read by row."""
    rng = np.random.default_rng(3)
    n = 200_000
    rk = rng.permutation(n).astype(np.int64)
    code = rng.integers(0, 200, n).astype(np.int32)
    if outlier:
        code[rk == n - 1] = np.iinfo(np.int32).min
    y = rng.integers(0, 9, n)
    lk = rng.integers(0, n - 1, 300_001).astype(np.int64)
    right = [make_column("rk", T.INT64, rk), make_column("code", T.INT32, code)] + ([make_column("y", T.INT64, y)] if extra else [])
    plan = make_group_by(["code"], [make_aggregate(A.COUNT_STAR, "", T.INT64)] + ([make_aggregate(A.MAX, "y", T.INT64)] if extra else []),
                         make_join("lk", "rk", ["code"] + (["y"] if extra else []), make_scan(["lk"]), make_scan([c.name for c in right])))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("lk", T.INT64, lk)] + right)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    assert "vgpu_gb_direct" in names and ("vgpu_stats" in names) == outlier, names
    at = np.argsort(rk)[lk]
    keys, counts = np.unique(code[at], return_counts=True)
    assert np.array_equal(r.columns[0].data, keys) and np.array_equal(r.columns[1].data, counts)
