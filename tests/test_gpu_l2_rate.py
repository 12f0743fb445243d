"""Which group-bys take the table in L2, on the B200: many state words over many rows are left to the partitioned passes,
the sooner the fewer slots their reductions meet in; results the same either way."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_aggregate, make_column, make_group_by, make_scan
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, hugeint_to_int, profile_drain, profile_enable

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,span,words,taken", [
    (1 << 20, 1 << 12, 7, True), ((1 << 20) + 1, 1 << 12, 7, False), (3_000_000, 1 << 17, 2, True), (3_000_000, 1 << 14, 2, True),
    (3_000_000, 1 << 15, 7, True), (3_000_000, 1 << 14, 7, False), (1_500_000, 1 << 18, 9, True), (1_800_000, 1 << 18, 9, False),
    (8_500_000, 1 << 23, 2, True), (8_500_000, 1 << 22, 3, False)])
def test_rows_words_and_slots(rows, span, words, taken):
    rng = np.random.default_rng(rows)
    k = rng.integers(0, span, rows).astype(np.int32)
    k[:2] = [0, span - 1]
    v = rng.integers(-(1 << 40), 1 << 40, rows)
    # a count and: nothing more / a 128-bit sum (two words) / MAX and MIN each
    aggs = [make_aggregate(A.MAX, "v", T.INT64)]
    if words == 3:
        aggs += [make_aggregate(A.MIN, "v", T.INT64)]
    elif words > 3:
        aggs += [make_aggregate(A.SUM, "v", T.HUGEINT)] + [make_aggregate(A.MIN, "v", T.INT64)] * (words - 4)
    plan = make_group_by(["k"], aggs, make_scan(["k", "v"]))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("k", T.INT32, k), make_column("v", T.INT64, v)])
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    assert ("vgpu_gb_l2" in names) == taken, names
    order = np.argsort(r.columns[0].data)
    by_key = np.lexsort((v, k))
    last = np.flatnonzero(np.diff(np.concatenate([k[by_key], [-1]])))
    first = np.concatenate([[0], last[:-1] + 1])
    assert np.array_equal(r.columns[0].data[order], k[by_key][last]) and np.array_equal(r.columns[1].data[order], v[by_key][last])
    if words == 3:
        assert np.array_equal(r.columns[2].data[order], v[by_key][first])
    elif words > 3:
        sums = np.add.reduceat(v[by_key], first)  # below 2^63: at most some 2^10 rows of 2^40
        assert hugeint_to_int(r.columns[2].data[order]) == sums.tolist()
