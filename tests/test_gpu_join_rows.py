"""The materializing join's tiled form on the B200 against numpy: left-major pairs, each left row's matches in
right row order, for every key width, repeats on either side of the run sorts' sizes, sparse keys, no matches,
rows around the tile size, and skew that leaves it to the balanced expansion."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_column, make_join, make_scan
from vectisdb_b200.engine import GpuValueType as T, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
NP = {T.BOOLEAN: np.uint8, T.INT16: np.int16, T.INT32: np.int32, T.INT64: np.int64}


def _join(lk, rk, kt, extra=()):
    rng = np.random.default_rng(1)
    a = rng.standard_normal(len(lk))
    b = rng.integers(-30_000, 30_000, len(rk)).astype(np.int16)
    c = rng.integers(0, 2, len(rk)).astype(np.uint8)
    d = rng.standard_normal(len(rk)).astype(np.float32)
    plan = make_join("lk", "rk", ["b", "lk", "a", "c", "d"], make_scan(["lk", "a"]), make_scan(["rk", "b", "c", "d"]))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [
            make_column("lk", kt, lk), make_column("a", T.FLOAT64, a), make_column("rk", kt, rk),
            make_column("b", T.INT16, b), make_column("c", T.BOOLEAN, c), make_column("d", T.FLOAT32, d)])
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    order = np.argsort(rk, kind="stable")
    first = np.searchsorted(rk[order], lk, side="left")
    count = np.searchsorted(rk[order], lk, side="right") - first
    left = np.repeat(np.arange(len(lk)), count)
    right = order[first[left] + np.arange(len(left)) - np.repeat(np.cumsum(count) - count, count)]
    for got, want in zip(r.columns, (b[right], lk[left], a[left], c[right], d[right])):
        assert got.data.dtype == want.dtype and np.array_equal(got.data, want), got.name
    return names


@pytest.mark.parametrize("left", [1, 255, 1023, 1024, 1025, 200_003])
def test_left_rows_around_the_tile_size(left):
    rng = np.random.default_rng(left)
    names = _join(rng.integers(-50, 5050, left).astype(np.int64), rng.integers(0, 5000, 9001).astype(np.int64), T.INT64)
    assert "join_emit" in names and "radix_scatter" not in names and "join_expand" not in names, names


@pytest.mark.parametrize("repeat,form", [(1, "join_emit"), (2, "join_emit"), (16, "join_emit"), (17, "join_emit"),
                                         (64, "join_emit"), (100, "join_expand")])
def test_repeats_of_every_key(repeat, form):
    """16 and 17 part the two run sorts; 64 matches a row fill the most a tile may have, 100 do not fit."""
    rng = np.random.default_rng(repeat)
    rk = np.repeat(rng.permutation(900).astype(np.int32) - 450, repeat)[rng.permutation(900 * repeat)]
    names = _join(rng.integers(-450, 450, 3000).astype(np.int32), rk, T.INT32)
    assert form in names, names


@pytest.mark.parametrize("longest,sorted_", [(4096, False), (4097, True)])
def test_one_long_run_met_by_few_left_rows(longest, sorted_):
    """Runs up to 4096 rows are put in order by one CTA; a longer one is sorted with the rest of the keys."""
    rng = np.random.default_rng(longest)
    rk = np.concatenate([np.full(longest, 5), rng.integers(6, 9000, 9000)]).astype(np.int64)[rng.permutation(longest + 9000)]
    lk = rng.integers(6, 9000, 50_000).astype(np.int64)
    lk[[3, 30_000]] = 5
    names = _join(lk, rk, T.INT64)
    assert ("radix_scatter" in names) == sorted_, names


@pytest.mark.parametrize("kt,lo,hi", [(T.BOOLEAN, 0, 2), (T.INT16, 10, 20_000), (T.INT64, 0, 1 << 50), (T.INT64, -(1 << 50), 1 << 50)])
def test_key_widths_and_sparse_keys(kt, lo, hi):
    rng = np.random.default_rng(hi % 1000)
    n = 40 if kt == T.BOOLEAN else 30_000
    rk = rng.integers(lo, hi, n).astype(NP[kt])
    lk = np.concatenate([rk[rng.integers(0, n, 5000 if n > 40 else 900)], rng.integers(lo, hi, 5000 if n > 40 else 9).astype(NP[kt])])
    names = _join(lk, np.concatenate([rk, rk[:10]]), kt)
    assert "join_emit" in names, names


def test_no_match_and_a_hot_left_key():
    rng = np.random.default_rng(4)
    _join(np.arange(100, 5000, dtype=np.int64), np.arange(0, 90, dtype=np.int64), T.INT64)
    lk = np.where(rng.random(60_000) < 0.5, 7, rng.integers(0, 3000, 60_000)).astype(np.int64)
    rk = np.concatenate([np.full(150, 7), rng.integers(0, 3000, 3000)]).astype(np.int64)
    names = _join(lk, rk, T.INT64)  # 512 rows of a tile with 150 matches each: past a tile's most
    assert "join_expand" in names, names


@pytest.mark.parametrize("spread", [1, 1 << 30])
@pytest.mark.parametrize("left,ordered", [((1 << 20) - 1, False), (1 << 20, True), ((1 << 20) + 77, True)])
def test_right_columns_in_run_order_from_four_matches_a_row(left, ordered, spread):
    """Four matches a right row and a million of them: the right columns are gathered into run order first."""
    rng = np.random.default_rng(9)
    rk = rng.permutation(1 << 18).astype(np.int64) * spread
    names = _join(rng.integers(0, 1 << 18, left).astype(np.int64) * spread, rk, T.INT64)
    assert ("gather" in names) == ordered and "join_emit" in names, names
