"""The one-pass group-by into a table that L2 holds, on the B200, against numpy: every aggregate kind over
skewed, sorted, constant and uniform keys, 64- and 128-bit integer sums on either side of the bound, key
spaces at both ends of its range, filters that keep nothing, join sources, and results whose count stays on
the device."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, device_to_host, make_aggregate,
                           make_column, make_expr, make_filter, make_group_by, make_join, make_scan)
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, hugeint_to_int, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
KERNEL = "vgpu_gb_l2"


def _run(plan, inputs, options=None):
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, inputs, options)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    assert KERNEL in names, names
    return r.columns


def _keys(kind, rng, n, base, span):
    if kind == "uniform":
        k = rng.integers(0, span, n)
    elif kind == "sorted":
        k = np.sort(rng.integers(0, span, n))
    elif kind == "constant":
        k = np.full(n, span // 3)
    else:  # most rows on few keys
        k = np.where(rng.random(n) < 0.7, rng.zipf(1.6, n) % span, rng.integers(0, span, n))
    k[0], k[-1] = 0, span - 1
    return k + base


@pytest.mark.parametrize("n", [2, 8191, 8192, 100_003, 1_500_001])
@pytest.mark.parametrize("kind", ["uniform", "sorted", "constant", "skewed"])
def test_every_aggregate_over_every_key_distribution(kind, n):
    rng = np.random.default_rng(n)
    k = _keys(kind, rng, n, -70_000, 150_000).astype(np.int32)
    v = rng.integers(-(1 << 62), 1 << 62, n, dtype=np.int64)  # sums need 128 bits
    s = rng.integers(-(1 << 31), 1 << 31, n, dtype=np.int64).astype(np.int32)  # sums fit 64
    x = rng.integers(-(1 << 20), 1 << 20, n).astype(np.float64)  # whole numbers: exact in any order
    f = rng.integers(-100, 100, n).astype(np.float32)
    cols = [make_column("k", T.INT32, k), make_column("v", T.INT64, v), make_column("s", T.INT32, s),
            make_column("x", T.FLOAT64, x), make_column("f", T.FLOAT32, f)]
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT), make_aggregate(A.SUM, "s", T.HUGEINT),
                                 make_aggregate(A.AVG, "s", T.FLOAT64), make_aggregate(A.SUM, "x", T.FLOAT64),
                                 make_aggregate(A.AVG, "f", T.FLOAT64), make_aggregate(A.MIN, "v", T.INT64),
                                 make_aggregate(A.MAX, "s", T.INT32), make_aggregate(A.COUNT_STAR, "", T.INT64)][2 * (n == 8192):],
                         make_scan(["k", "v", "s", "x", "f"]))
    got = _run(plan, cols)
    keys, inv = np.unique(k, return_inverse=True)
    count = np.bincount(inv)
    assert np.array_equal(got[0].data, keys)  # in key order
    if n != 8192:
        exp_v, exp_s = [0] * len(keys), [0] * len(keys)
        for i, a, b in zip(inv.tolist(), v.tolist(), s.tolist()):
            exp_v[i] += a
            exp_s[i] += b
        assert hugeint_to_int(got[1].data) == exp_v and hugeint_to_int(got[2].data) == exp_s
    got = got[-6:]
    assert np.array_equal(got[0].data, np.bincount(inv, weights=s.astype(np.float64)) / count)
    assert np.array_equal(got[1].data, np.bincount(inv, weights=x))
    assert np.array_equal(got[2].data, np.bincount(inv, weights=f.astype(np.float64)) / count)
    lo, hi = np.full(len(keys), np.iinfo(np.int64).max), np.full(len(keys), np.iinfo(np.int32).min)
    np.minimum.at(lo, inv, v)
    np.maximum.at(hi, inv, s)
    assert np.array_equal(got[3].data, lo) and np.array_equal(got[4].data, hi) and np.array_equal(got[5].data, count)


@pytest.mark.parametrize("limit", [1 << 30, (1 << 63) // 400_003, (1 << 63) // 400_003 + 1, (1 << 62)])
def test_cached_integer_sums_on_either_side_of_64_bits(limit):
    """The cached column's range decides whether a sum keeps one 64-bit word: totals at and past the bound."""
    n = 400_003
    rng = np.random.default_rng(1)
    k = rng.integers(0, 30_000, n).astype(np.int32)
    k[: n // 2] = 7  # half the rows, all of the largest value, on one key
    v = rng.integers(-limit, limit, n, dtype=np.int64)
    v[: n // 2] = limit
    ref = GpuTableRef("memory", "main", "l2sums")
    ColumnCache.put_table(ref, [make_column("k", T.INT32, k), make_column("v", T.INT64, v)])
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT)], make_scan(["k", "v"], ref))
    try:
        got = _run(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True))
    finally:
        ColumnCache.invalidate_table(ref)
    exp = {}
    for key, x in zip(k.tolist(), v.tolist()):
        exp[key] = exp.get(key, 0) + x
    assert dict(zip(got[0].data.tolist(), hugeint_to_int(got[1].data))) == exp


@pytest.mark.parametrize("span,taken", [(12_288, False), (12_289, True), (1 << 23, True), ((1 << 23) + 1, True)])
def test_range_of_key_spaces(span, taken):
    """COUNT(*) alone: one state word per slot, so 2^13 slots still fit shared memory and 2^23 make 64 MB;
    past that few rows of many key values are hashed."""
    span = {12_288: 8192, 12_289: 16_384}.get(span, span)
    rng = np.random.default_rng(span)
    k = rng.integers(0, span, 300_000).astype(np.int32)
    k[:2] = [0, span - 1]
    plan = make_group_by(["k"], [make_aggregate(A.COUNT_STAR, "", T.INT64)], make_scan(["k"]))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("k", T.INT32, k)])
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success and (KERNEL in names) == taken, names
    keys, counts = np.unique(k, return_counts=True)
    order = np.argsort(r.columns[0].data)
    assert np.array_equal(r.columns[0].data[order], keys) and np.array_equal(r.columns[1].data[order], counts)


def test_two_keys_a_filter_that_keeps_nothing_and_counts_left_on_the_device():
    import torch
    rng = np.random.default_rng(9)
    n = 200_003
    a = rng.integers(-50, 350, n).astype(np.int16)
    b = rng.integers(1000, 1100, n).astype(np.int64)
    x = rng.integers(0, 1000, n).astype(np.float64)
    ref = GpuTableRef("memory", "main", "l2two")
    ColumnCache.put_table(ref, [make_column("a", T.INT16, a), make_column("b", T.INT64, b), make_column("x", T.FLOAT64, x)])
    stream = torch.cuda.Stream().cuda_stream
    lazy = ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True, no_sync=True, stream=stream)

    def plan(bound):
        filt = make_filter([make_expr(f"((bool*)out)[idx] = ((const double*)inputs[0])[row] < {bound}.0;", ["x"], T.BOOLEAN)],
                           make_scan(["a", "b", "x"], ref))
        return make_group_by(["a", "b"], [make_aggregate(A.SUM, "x", T.FLOAT64)], filt)
    try:
        queued = [GpuEngine.instance().execute_plan(plan(w), [], lazy) for w in (500, 0, 1000)]
        for w, r in zip((500, 0, 1000), queued):
            keep = x < w
            packed = a[keep].astype(np.int64) * 10_000 + b[keep]
            keys, inv = np.unique(packed, return_inverse=True)
            got = [device_to_host(c, stream) for c in r.columns]
            r.free()
            got_key = got[0].astype(np.int64) * 10_000 + got[1]
            order = np.argsort(got_key)
            assert np.array_equal(got_key[order], keys)
            assert np.array_equal(got[2][order], np.bincount(inv, weights=x[keep], minlength=len(keys)))
    finally:
        ColumnCache.invalidate_table(ref)


@pytest.mark.parametrize("repeat", [1, 3])
def test_over_a_join_with_one_and_several_matches(repeat):
    rng = np.random.default_rng(repeat)
    rk = np.repeat(rng.permutation(60_000).astype(np.int64), repeat)
    rg = rng.integers(0, 200_000, len(rk)).astype(np.int32)
    lk = rng.integers(0, 70_000, 250_003).astype(np.int64)
    lv = rng.integers(-1000, 1000, len(lk)).astype(np.int64)
    plan = make_group_by(["rg"], [make_aggregate(A.SUM, "lv", T.HUGEINT), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_join("lk", "rk", ["rg", "lv"], make_scan(["lk", "lv"]), make_scan(["rk", "rg"])))
    got = _run(plan, [make_column("lk", T.INT64, lk), make_column("lv", T.INT64, lv), make_column("rk", T.INT64, rk),
                      make_column("rg", T.INT32, rg)])
    first = np.full(70_000, -1)
    order = np.argsort(rk, kind="stable")
    first[rk[order][::repeat]] = np.arange(60_000) * repeat
    hit = first[lk] >= 0
    left = np.repeat(np.flatnonzero(hit), repeat)
    g = rg[order][(first[lk[hit]][:, None] + np.arange(repeat)).ravel()]
    keys, inv = np.unique(g, return_inverse=True)
    assert np.array_equal(got[0].data, keys)
    assert hugeint_to_int(got[1].data) == np.bincount(inv, weights=lv[left]).astype(np.int64).tolist()
    assert np.array_equal(got[2].data, np.bincount(inv))


@pytest.mark.parametrize("n,distinct,bits", [(2, 2, 62), (1000, 1000, 40), (8192, 3000, 63), (300_007, 60_000, 50),
                                             (1_000_003, 1_000_003, 60), (2_000_003, 700_001, 55)])
def test_sparse_keys_in_a_hashed_table(n, distinct, bits):
    rng = np.random.default_rng(n)
    ids = np.unique(np.concatenate([[0, (1 << bits) - 1], rng.integers(0, 1 << bits, distinct, dtype=np.int64)]))
    pick = rng.integers(0, len(ids), n) if distinct < n else rng.permutation(np.arange(n) % len(ids))
    hot = rng.random(n) < 0.3
    pick[hot & (distinct < n)] = 1  # a frequent key
    pick[:2] = [0, len(ids) - 1]
    k = ids[pick] - (1 << 40)
    v = rng.integers(-(1 << 62), 1 << 62, n, dtype=np.int64)
    x = rng.integers(-1000, 1000, n).astype(np.float64)
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "x", T.FLOAT64), make_aggregate(A.MIN, "v", T.INT64),
                                 make_aggregate(A.COUNT_STAR, "", T.INT64)], make_scan(["k", "x", "v"]))
    got = _run(plan, [make_column("k", T.INT64, k), make_column("x", T.FLOAT64, x), make_column("v", T.INT64, v)])
    keys, inv = np.unique(k, return_inverse=True)
    order = np.argsort(got[0].data)
    assert np.array_equal(got[0].data[order], keys)
    assert np.array_equal(got[1].data[order], np.bincount(inv, weights=x))
    lo = np.full(len(keys), np.iinfo(np.int64).max)
    np.minimum.at(lo, inv, v)
    assert np.array_equal(got[2].data[order], lo) and np.array_equal(got[3].data[order], np.bincount(inv))


@pytest.mark.parametrize("keys,estimate,tried", [("pairs", 0, True), ("pairs", 600_000, True), ("pairs", 700_000, False),
                                                 ("one", 0, False)])
def test_more_sparse_keys_than_the_hashed_table_holds(keys, estimate, tried):
    """Seven state words and the key make 2^20 slots of 64 MB. 1.5M pairs of two keys with some 1200 values each
    end the pass, and the partitions do it; the plan's estimate, or one key's own distinct count, says so before."""
    rng = np.random.default_rng(3)
    n = 1_500_001
    order = rng.permutation(n).astype(np.int64)
    a, b = (order // 1225 * 1001, order % 1225 * 997) if keys == "pairs" else (order * 1_000_003, np.zeros(n, np.int64))
    cols = [make_column("a", T.INT64, a), make_column("b", T.INT64, b)]
    cols += [make_column(f"x{i}", T.INT64, np.roll(order, i + 1)) for i in range(6)]
    plan = make_group_by(["a", "b"], [make_aggregate(A.MAX, f"x{i}", T.INT64) for i in range(6)],
                         make_scan([c.name for c in cols]))
    plan.estimated_rows = estimate
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, cols)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success and (KERNEL in names) == tried and "vgpu_gb_bucket" in names, names
    got, want = np.lexsort((r.columns[1].data, r.columns[0].data)), np.lexsort((b, a))
    assert np.array_equal(r.columns[0].data[got], a[want]) and np.array_equal(r.columns[1].data[got], b[want])
    for i in range(6):
        assert np.array_equal(r.columns[2 + i].data[got], cols[2 + i].data[want])


@pytest.mark.parametrize("n,taken", [((1 << 23) - 1, False), (1 << 23, True)])
def test_tables_of_128_megabytes_from_a_row_for_each_slot(n, taken):
    rng = np.random.default_rng(21)
    k = (rng.integers(0, 1 << 23, n) - 999).astype(np.int32)
    k[0], k[-1] = -999, (1 << 23) - 1000
    v = rng.integers(-1000, 1000, n).astype(np.int32)
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["k", "v"]))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("k", T.INT32, k), make_column("v", T.INT32, v)])
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    assert (KERNEL in names) == taken and ("vgpu_gb_dbucket" in names) != taken, names
    at = k.astype(np.int64) + 999
    counts = np.bincount(at, minlength=1 << 23)
    sums = np.bincount(at, weights=v, minlength=1 << 23).astype(np.int64)  # exact: below 2^53
    got = r.columns[0].data.astype(np.int64) + 999
    order = np.argsort(got)
    assert np.array_equal(got[order], np.flatnonzero(counts))
    assert np.array_equal(r.columns[2].data[order], counts[counts > 0])
    assert np.array_equal(r.columns[1].data["lower"][order].view(np.int64), sums[counts > 0])
