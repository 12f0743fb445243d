"""The one-pass row filter on the B200 against the two-pass form and numpy: rows around the tile size, no,
all and few rows kept, rows too wide for its staging, nullable outputs, a join source and a cross product,
results that give back the room of the dropped rows, and plans whose estimate keeps the two-pass form."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, device_to_host, make_column,
                           make_cross_product, make_expr, make_filter, make_join, make_projection, make_scan)
from vectisdb_b200.engine import GpuValueType as T, memory_stats, profile_drain, profile_enable

pytestmark = pytest.mark.gpu

ROWS = [1, 2, 511, 512, 513, 1024, 1025, 65_535, 65_537, 1_000_003]


def _filter(bound, child, column="x"):
    return make_filter([make_expr(f"((bool*)out)[idx] = (((const int*)inputs[0])[row] < {bound});", [column], T.BOOLEAN)],
                       child)


def _launched(plan, inputs, options=None):
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, inputs, options)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    return r, names


def _both_forms(plan, inputs, monkeypatch):
    """Columns of the one-pass form, after checking that the two-pass form gives the same."""
    one, names = _launched(plan, inputs)
    assert one.success, one.error_message
    assert "vgpu_mat_onepass" in names and "vgpu_mat_count" not in names, names
    monkeypatch.setenv("VGPU_MAT_PASSES", "2")
    two, names = _launched(plan, inputs)
    monkeypatch.delenv("VGPU_MAT_PASSES")
    assert "vgpu_mat_onepass" not in names and "vgpu_mat_count" in names, names
    for a, b in zip(one.columns, two.columns):
        assert a.row_count == b.row_count and a.data.tobytes() == b.data.tobytes(), a.name
        assert (a.validity is None) == (b.validity is None)
        assert a.validity is None or np.array_equal(a.validity, b.validity)
    return one.columns


@pytest.mark.parametrize("bound", [0, 37, 100])  # of 100 values: no, some, all rows kept
@pytest.mark.parametrize("rows", ROWS)
def test_rows_around_the_tile_size(rows, bound, monkeypatch):
    rng = np.random.default_rng(rows + bound)
    x = rng.integers(0, 100, rows).astype(np.int32)
    b = (x % 2).astype(np.uint8)
    s = rng.integers(-30_000, 30_000, rows).astype(np.int16)
    d = rng.standard_normal(rows)
    cols = [make_column("x", T.INT32, x), make_column("b", T.BOOLEAN, b), make_column("s", T.INT16, s),
            make_column("d", T.FLOAT64, d)]
    got = _both_forms(_filter(bound, make_scan(["x", "b", "s", "d"])), cols, monkeypatch)
    keep = x < bound
    for c, v in zip(got, (x, b, s, d)):
        assert np.array_equal(c.data, v[keep]), c.name


@pytest.mark.parametrize("rows", [513, 200_003])
def test_nullable_columns(rows, monkeypatch):
    rng = np.random.default_rng(rows)
    x = rng.integers(0, 100, rows).astype(np.int32)
    y = rng.integers(-(1 << 40), 1 << 40, rows).astype(np.int64)
    xv, yv = rng.random(rows) < 0.9, rng.random(rows) < 0.6
    cols = [make_column("x", T.INT32, x, xv), make_column("y", T.INT64, y, yv)]
    got = _both_forms(_filter(60, make_scan(["x", "y"])), cols, monkeypatch)
    keep = (x < 60) & xv
    assert np.array_equal(got[0].data, x[keep])
    assert np.array_equal(got[1].validity, yv[keep])
    assert np.array_equal(got[1].data[yv[keep]], y[keep & yv])


def test_join_source_and_cross_product(monkeypatch):
    rng = np.random.default_rng(3)
    rk = rng.permutation(5000).astype(np.int64)
    rv = rng.integers(0, 100, 5000).astype(np.int32)
    lk = rng.integers(-100, 6000, 100_001).astype(np.int64)
    lv = rng.standard_normal(len(lk))
    join = make_join("lk", "rk", ["lv", "rv"], make_scan(["lk", "lv"]), make_scan(["rk", "rv"]))
    got = _both_forms(_filter(50, join, "rv"), [make_column("lk", T.INT64, lk), make_column("lv", T.FLOAT64, lv),
                                               make_column("rk", T.INT64, rk), make_column("rv", T.INT32, rv)], monkeypatch)
    pos = np.full(6000, -1)
    pos[rk] = np.arange(5000)
    hit = np.where((lk >= 0), pos[np.clip(lk, 0, 5999)], -1)
    keep = (hit >= 0) & (rv[hit] < 50)
    assert np.array_equal(got[0].data, lv[keep]) and np.array_equal(got[1].data, rv[hit[keep]])
    a, b = rng.integers(0, 100, 701).astype(np.int32), rng.integers(0, 100, 903).astype(np.int32)
    cross = make_cross_product(["a", "b"], make_scan(["a"]), make_scan(["b"]))
    got = _both_forms(_filter(7, cross, "a"), [make_column("a", T.INT32, a), make_column("b", T.INT32, b)], monkeypatch)
    la, lb = np.repeat(a, len(b)), np.tile(b, len(a))
    assert np.array_equal(got[0].data, la[la < 7]) and np.array_equal(got[1].data, lb[la < 7])


@pytest.mark.parametrize("columns,one_pass", [(11, True), (12, False)])  # 92 and 100 bytes a row
def test_wide_rows(columns, one_pass):
    rng = np.random.default_rng(columns)
    n = 30_011
    x = rng.integers(0, 100, n).astype(np.int32)
    ys = [rng.integers(-(1 << 60), 1 << 60, n).astype(np.int64) for _ in range(columns)]
    cols = [make_column("x", T.INT32, x)] + [make_column(f"y{i}", T.INT64, y) for i, y in enumerate(ys)]
    r, names = _launched(_filter(42, make_scan([c.name for c in cols])), cols)
    assert r.success and ("vgpu_mat_onepass" in names) == one_pass, names
    for c, v in zip(r.columns, [x] + ys):
        assert np.array_equal(c.data, v[x < 42]), c.name


@pytest.mark.parametrize("estimate,one_pass", [(0, True), (2_000_000, True), (1_000_000, False)])
def test_the_plans_estimate_keeps_the_two_pass_form(estimate, one_pass):
    n = 4_000_000
    x = (np.arange(n) % 100).astype(np.int32)
    plan = _filter(50, make_scan(["x"]))
    plan.estimated_rows = estimate
    r, names = _launched(plan, [make_column("x", T.INT32, x)])
    assert r.success and ("vgpu_mat_onepass" in names) == one_pass, names
    assert np.array_equal(r.columns[0].data, x[x < 50])


@pytest.mark.parametrize("bound,held", [(5, 0.06), (60, 1.01)])
def test_a_result_of_few_rows_gives_the_room_back(bound, held):
    n = 12_000_000  # 8 + 4 bytes a row: 144 MB if every row were kept
    x = (np.arange(n) % 100).astype(np.int32)
    ref = GpuTableRef("memory", "main", "onepass_room")
    ColumnCache.put_table(ref, [make_column("x", T.INT32, x), make_column("d", T.FLOAT64, np.arange(n, dtype=np.float64))])
    plan = make_projection([make_expr("((int*)out)[idx] = ((const int*)inputs[0])[row];", ["x"], T.INT32),
                            make_expr("((double*)out)[idx] = ((const double*)inputs[0])[row] + 1.0;", ["d"], T.FLOAT64)],
                           _filter(bound, make_scan(["x", "d"], ref)))
    try:
        before = memory_stats()["in_use_bytes"]
        r = GpuEngine.instance().execute_plan(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True))
        used = memory_stats()["in_use_bytes"] - before
        got = [device_to_host(c) for c in r.columns]
        r.free()
        assert used <= held * n * 12, used
        assert np.array_equal(got[0], x[x < bound]) and np.array_equal(got[1], np.flatnonzero(x < bound) + 1.0)
        assert memory_stats()["in_use_bytes"] == before
    finally:
        ColumnCache.invalidate_table(ref)
