"""Value ranges read from whole columns and the dense join tables built on them, on the B200: columns that
start off a 16-byte boundary, lengths around the vector and CTA sizes, extreme values at either end, every
key and value width, and right sides whose only repeated key is the last row."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from vectisdb_b200 import GpuEngine, make_aggregate, make_group_by, make_join, make_scan
from vectisdb_b200.engine import (GpuAggregateKind as A, GpuTableRef, GpuValueType as T, make_device_column,
                                  hugeint_to_int)

pytestmark = pytest.mark.gpu

NP = {T.INT16: np.int16, T.INT32: np.int32, T.INT64: np.int64, T.BOOLEAN: np.uint8}


def _on_device(name, t, values, skip):
    """A device column over values[skip:] of a device array: its address is off the allocation's by skip."""
    dev = torch.from_numpy(np.ascontiguousarray(values)).cuda()
    return make_device_column(name, t, dev.data_ptr() + skip * dev.element_size(), len(values) - skip), dev


def _run(plan, columns):
    torch.cuda.synchronize()
    r = GpuEngine.instance().execute_plan(plan, columns)
    assert r.success, r.error_message
    return r.columns


@pytest.mark.parametrize("skip", [0, 1, 3])
@pytest.mark.parametrize("rows", [1, 2, 15, 17, 4095, 70_001, 1_200_007])
@pytest.mark.parametrize("t", [T.BOOLEAN, T.INT16, T.INT32, T.INT64])
def test_group_by_key_range_of_device_columns(t, rows, skip):
    rng = np.random.default_rng(rows * 7 + skip)
    base = {T.BOOLEAN: 0, T.INT16: -30_000, T.INT32: -2_000_000_000, T.INT64: -(1 << 62)}[t]
    span = 2 if t == T.BOOLEAN else 700
    k = (base + rng.integers(0, span, rows + skip)).astype(NP[t])
    k[skip] = base + span - 1  # the extremes sit in the first and last rows
    k[-1] = base
    col, keep = _on_device("k", t, k, skip)
    plan = make_group_by(["k"], [make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["k"], GpuTableRef("memory", "main", "bounds")))
    got = _run(plan, [col])
    keys, counts = np.unique(k[skip:], return_counts=True)
    assert np.array_equal(got[0].data, keys) and np.array_equal(got[1].data, counts)
    del keep


@pytest.mark.parametrize("repeated", [False, True])
@pytest.mark.parametrize("kt,vt,rows", [(T.INT16, T.INT16, 3001), (T.INT32, T.INT32, 40_003), (T.INT64, T.INT16, 65_537),
                                        (T.INT64, T.BOOLEAN, 1021), (T.INT32, T.INT64, 9_999)])
def test_dense_table_of_every_key_and_value_width(kt, vt, rows, repeated):
    rng = np.random.default_rng(rows)
    rk = (5 + rng.permutation(rows)).astype(NP[kt])
    rg = rng.integers(-120 if vt != T.BOOLEAN else 0, 120 if vt != T.BOOLEAN else 2, rows).astype(NP[vt])
    if repeated:
        rk[-1] = rk[1]  # one entry short: not a unique-key table
    lk = rng.integers(0, rows + 50, 100_003).astype(NP[kt])
    lv = rng.integers(-1000, 1000, len(lk)).astype(np.int64)
    cols, keep = zip(*[_on_device(n, t, v, 1) for n, t, v in
                       [("lk", kt, lk), ("lv", T.INT64, lv), ("rk", kt, rk), ("rg", vt, rg)]])
    plan = make_group_by(["rg"], [make_aggregate(A.SUM, "lv", T.HUGEINT), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_join("lk", "rk", ["rg", "lv"], make_scan(["lk", "lv"], GpuTableRef("memory", "main", "bl")),
                                   make_scan(["rk", "rg"], GpuTableRef("memory", "main", "br"))))
    got = _run(plan, list(cols))
    lk, lv, rk, rg = lk[1:], lv[1:], rk[1:], rg[1:]  # skip = 1
    per_key = {}
    for key, g in zip(rk.tolist(), rg.tolist()):
        per_key.setdefault(key, []).append(g)
    sums, counts = {}, {}
    for key, v in zip(lk.tolist(), lv.tolist()):
        for g in per_key.get(key, ()):
            sums[g] = sums.get(g, 0) + v
            counts[g] = counts.get(g, 0) + 1
    have = dict(zip(got[0].data.tolist(), zip(hugeint_to_int(got[1].data), got[2].data.tolist())))
    assert have == {g: (sums[g], counts[g]) for g in counts}
    del keep
