"""The materializing join over uneven right sides on the B200, against numpy: half of the rows on one key, runs around the
sizes where their sort changes hands, left rows with thousands of matches each, and a hot left key whose matches are
expanded from the grouped rows."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_column, make_join, make_scan
from vectisdb_b200.engine import GpuValueType as T, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
KEYS = {T.INT16: np.int16, T.INT32: np.int32, T.INT64: np.int64}


def _join(lk, rk, kt=T.INT64):
    lk, rk = np.asarray(lk).astype(KEYS[kt]), np.asarray(rk).astype(KEYS[kt])
    b = np.arange(len(rk), dtype=np.int32)
    plan = make_join("lk", "rk", ["lk", "b"], make_scan(["lk"]), make_scan(["rk", "b"]))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("lk", kt, lk), make_column("rk", kt, rk), make_column("b", T.INT32, b)])
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    order = np.argsort(rk, kind="stable")
    first = np.searchsorted(rk[order], lk, side="left")
    count = np.searchsorted(rk[order], lk, side="right") - first
    left = np.repeat(np.arange(len(lk)), count)
    right = order[first[left] + np.arange(len(left)) - np.repeat(np.cumsum(count) - count, count)]
    assert np.array_equal(r.columns[0].data, lk[left]) and np.array_equal(r.columns[1].data, b[right])
    return names


@pytest.mark.parametrize("kt", [T.INT32, T.INT64])
@pytest.mark.parametrize("n,share", [(20_000, 0.5), (300_000, 0.5), (1_000_003, 0.9), (1_000_003, 0.02)])
def test_a_key_with_many_of_the_rows_is_sorted_at_once(n, share, kt):
    rng = np.random.default_rng(n)
    rk = np.where(rng.random(n) < share, 5, rng.integers(0, n, n))
    lk = rng.integers(6, n, 3000)
    lk[7] = 5
    names = _join(lk, rk, kt)
    assert "radix_scatter" in names and "join_runs_dense" not in names, names


@pytest.mark.parametrize("length", [15, 16, 17, 31, 32, 33, 63, 65, 255, 256, 257, 300, 1500])
def test_runs_around_the_sizes_of_their_sorts(length):
    rng = np.random.default_rng(length)
    rk = np.concatenate([np.repeat(rng.integers(0, 15_000, 9), length), np.repeat(20, length), np.arange(15_000)])
    names = _join(rng.integers(0, 15_000, 2000), rng.permutation(rk))
    assert "join_runs_dense" in names and "radix_scatter" not in names, names


def test_equal_neighbours_in_every_warp():
    """Right keys in order, so that neighbours share their key, in blocks of one to seven, and the last one alone."""
    rk = np.repeat(np.arange(30_000), np.arange(30_000) % 7 + 1)
    for cut in (0, 1, 31, 32):
        names = _join(np.arange(-5, 30_010, 3), rk[: len(rk) - cut])
        assert "join_runs_dense" in names, names


@pytest.mark.parametrize("left,matches", [(1, 3000), (300, 64), (600, 100), (750, 80), (1024, 63), (2000, 60)])
def test_few_left_rows_with_many_matches(left, matches):
    """One tile's matches are shared by several CTAs."""
    rng = np.random.default_rng(matches)
    rk = np.concatenate([np.repeat(np.arange(left) * 3, matches), 3 * left + np.arange(4 * matches)])
    names = _join(np.arange(left) * 3, rng.permutation(rk), T.INT32)
    assert "join_emit" in names, names


@pytest.mark.parametrize("sparse", [False, True])
def test_a_hot_left_key_is_expanded_from_the_grouped_rows(sparse):
    rng = np.random.default_rng(1)
    step = 1 << 33 if sparse else 1
    rk = np.concatenate([np.full(200, 7), np.arange(40_000)])
    lk = np.where(rng.random(30_000) < 0.5, 7, rng.integers(0, 40_000, 30_000))
    names = _join(lk * step, rng.permutation(rk) * step)
    assert "join_expand" in names and ("radix_scatter" in names) == sparse, names
