"""BOOLEAN columns whose true values are other bytes than 1, on the B200, cached (so that their ranges are known) and
not: as join keys, matched by the byte, and as the value that a join's table holds."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column,
                           make_group_by, make_join, make_scan)
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
