"""BOOLEAN columns whose true values are other bytes than 1, on the B200, cached (so that their ranges are known) and
not: as join keys, matched by the byte, as the value that a join's table holds, and as group keys, where any byte
but 0 is true, read in whole vectors, row by row, from a join's right side and from a cross product."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column,
                           make_cross_product, make_group_by, make_join, make_scan)
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T

pytestmark = pytest.mark.gpu


def _run(plan, tables, cached):
    """`plan` of the tables' references; each table a name -> columns."""
    refs = {name: GpuTableRef("memory", "main", "bytes_" + name) for name in tables}
    try:
        if cached:
            for name, cols in tables.items():
                ColumnCache.put_table(refs[name], cols)
        r = GpuEngine.instance().execute_plan(plan(refs), [] if cached else [c for cols in tables.values() for c in cols],
                                              ExecuteOptions(serve_whole_scan_from_cache=cached))
    finally:
        for ref in refs.values():
            ColumnCache.invalidate_table(ref)
    assert r.success, r.error_message
    return [c.data for c in r.columns]


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("right", [[1], [255], [0, 255], [255, 1, 0], [0, 1, 2, 255, 255, 128], [3, 3, 3, 200]])
def test_join_keys_match_by_the_byte(right, cached):
    left = (np.arange(1000) % 3 == 0).astype(np.uint8)
    group = (np.arange(len(right)) * 3).astype(np.int32)
    tables = {"left": [make_column("lk", T.BOOLEAN, left)],
              "right": [make_column("rk", T.BOOLEAN, right), make_column("g", T.INT32, group)]}
    got = _run(lambda t: make_group_by(["g"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                                       make_join("lk", "rk", ["g"], make_scan(["lk"], t["left"]),
                                                 make_scan(["rk", "g"], t["right"]))), tables, cached)
    want = {int(g): int((left == r).sum()) for r, g in zip(right, group) if (left == r).any()}
    assert dict(zip(got[0].tolist(), got[1].tolist())) == want


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("repeat", [1, 2])
def test_values_held_in_the_joins_table(repeat, cached):
    rng = np.random.default_rng(repeat)
    rk = np.repeat(rng.permutation(3000).astype(np.int32), repeat)
    flag = rng.choice(np.array([0, 1, 2, 255], np.uint8), len(rk))
    lk = rng.integers(0, 3000, 20_001).astype(np.int32)
    tables = {"left": [make_column("lk", T.INT32, lk)],
              "right": [make_column("rk", T.INT32, rk), make_column("flag", T.BOOLEAN, flag)]}
    got = _run(lambda t: make_group_by(["flag"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                                       make_join("lk", "rk", ["flag"], make_scan(["lk"], t["left"]),
                                                 make_scan(["rk", "flag"], t["right"]))), tables, cached)
    true = np.bincount(rk, weights=flag != 0, minlength=3000)[lk].sum()
    assert got[0].tolist() == [0, 1] and got[1].tolist() == [len(lk) * repeat - true, true]


def _counts(flags):
    return [0, 1][int(flags.all()):2 if flags.any() else 1], [n for n in (int((flags == 0).sum()), int((flags != 0).sum())) if n]


def _flags(n):
    return np.random.default_rng(n).choice(np.array([0, 1, 2, 128, 255], np.uint8), n)


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4099, 700_001])
def test_group_keys(n, cached):
    flag = _flags(n)
    got = _run(lambda t: make_group_by(["flag"], [make_aggregate(A.COUNT_STAR, "", T.INT64)], make_scan(["flag"], t["t"])),
               {"t": [make_column("flag", T.BOOLEAN, flag)]}, cached)
    keys, counts = _counts(flag)
    assert got[0].tolist() == keys and got[1].tolist() == counts


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("repeat", [1, 2])
@pytest.mark.parametrize("side", ["left", "right"])
def test_group_keys_over_a_join(side, repeat, sparse, cached):
    """Two right columns, so that they are read at the match's row and not from the table of keys."""
    rk = np.repeat(np.arange(500, dtype=np.int64) * (1 << 33 if sparse else 1), repeat)
    lk = rk[:: repeat][np.random.default_rng(1).integers(0, 500, 3001)]
    left, right = _flags(len(lk)), _flags(len(rk))
    tables = {"left": [make_column("lk", T.INT64, lk), make_column("lf", T.BOOLEAN, left)],
              "right": [make_column("rk", T.INT64, rk), make_column("rf", T.BOOLEAN, right),
                        make_column("w", T.INT64, np.arange(len(rk)) % 5)]}
    key = side[0] + "f"
    got = _run(lambda t: make_group_by([key, "w"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                                       make_join("lk", "rk", ["lf", "rf", "w"], make_scan(["lk", "lf"], t["left"]),
                                                 make_scan(["rk", "rf", "w"], t["right"]))), tables, cached)
    first = np.searchsorted(rk, lk)
    want = {}
    for j in range(repeat):
        flags = left if side == "left" else right[first + j]
        for f, w in zip((flags != 0).tolist(), ((first + j) % 5).tolist()):
            want[(int(f), w)] = want.get((int(f), w), 0) + 1
    assert {(int(f), int(w)): int(c) for f, w, c in zip(*got)} == want


@pytest.mark.parametrize("cached", [False, True])
def test_group_keys_over_a_cross_product(cached):
    a, b = _flags(301), _flags(77)
    got = _run(lambda t: make_group_by(["a", "b"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                                       make_cross_product(["a", "b"], make_scan(["a"], t["left"]), make_scan(["b"], t["right"]))),
               {"left": [make_column("a", T.BOOLEAN, a)], "right": [make_column("b", T.BOOLEAN, b)]}, cached)
    want = {(f, g): int(((a != 0) == f).sum()) * int(((b != 0) == g).sum()) for f in (0, 1) for g in (0, 1)}
    assert {(int(f), int(g)): int(c) for f, g, c in zip(*got)} == want


def test_group_keys_of_the_partitioned_passes_over_staged_tiles():
    """A key of 2^22 values beside the flag: direct-partitioned, its count and scatter passes over staged tiles."""
    n = 3_000_000
    k = (np.arange(n, dtype=np.int64) * 2_654_435_761 % (1 << 22)).astype(np.int32)
    flag = _flags(n)
    cols = [make_column("k", T.INT32, k), make_column("flag", T.BOOLEAN, flag), make_column("v", T.INT64, np.ones(n)),
            make_column("x", T.FLOAT64, np.ones(n))]
    got = _run(lambda t: make_group_by(["k", "flag"], [make_aggregate(A.SUM, "v", T.HUGEINT), make_aggregate(A.MAX, "v", T.INT64),
                                                       make_aggregate(A.SUM, "x", T.FLOAT64)],
                                       make_scan(["k", "flag", "v", "x"], t["t"])), {"t": cols}, True)
    keys, counts = np.unique(k.astype(np.int64) * 2 + (flag != 0), return_counts=True)
    packed = got[0].astype(np.int64) * 2 + got[1]
    order = np.argsort(packed)
    assert np.array_equal(packed[order], keys) and np.array_equal(got[4][order], counts)
