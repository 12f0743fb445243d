"""Sparse keys of two columns on the B200, whose joint number no statistic tells: pairs that fit the hashed table in L2 and
pairs that do not, evenly spread and beside a frequent one, and filters that leave the sample little to go by."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_aggregate, make_column, make_expr, make_filter, make_group_by, make_scan
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
N = 2_000_003
SLOTS = 1 << 21  # of 24 bytes (key, SUM, COUNT) within 64 MB


@pytest.mark.parametrize("frequent", [0.0, 0.6])
@pytest.mark.parametrize("share,fits", [(0.001, True), (0.4, True), (0.85, False)])
@pytest.mark.parametrize("kept", [1000, 100, 2])
def test_pairs_that_fit_and_pairs_that_do_not(share, fits, frequent, kept):
    rng = np.random.default_rng(int(share * 1000))
    pairs = int(share * SLOTS)
    ids = rng.permutation(np.arange(N) % pairs)
    ids[rng.random(N) < frequent] = 0
    a, b = ids // 1500 * 10_007, ids % 1500 * 1_000_003
    x = (np.arange(N) % 1000).astype(np.float64)
    cols = [make_column("a", T.INT64, a), make_column("b", T.INT64, b), make_column("x", T.FLOAT64, x)]
    filt = make_filter([make_expr(f"((bool*)out)[idx] = ((const double*)inputs[0])[row] < {kept}.0;", ["x"], T.BOOLEAN)],
                       make_scan(["a", "b", "x"]))
    plan = make_group_by(["a", "b"], [make_aggregate(A.SUM, "x", T.FLOAT64), make_aggregate(A.COUNT_STAR, "", T.INT64)], filt)
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, cols)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    keep = x < kept
    keys, inv = np.unique(ids[keep], return_inverse=True)
    assert "vgpu_gb_l2_guess" in names, names
    if len(keys) < 0.5 * SLOTS or len(keys) > 0.75 * SLOTS:  # (between: either)
        assert ("vgpu_gb_bucket" in names) == (len(keys) > 0.75 * SLOTS), names
    assert kept < 1000 or frequent or (len(keys) > 0.75 * SLOTS) != fits
    got = r.columns[0].data // 10_007 * 1500 + r.columns[1].data // 1_000_003
    order = np.argsort(got)
    assert np.array_equal(got[order], keys)
    assert np.array_equal(r.columns[2].data[order], np.bincount(inv, weights=x[keep]))
    assert np.array_equal(r.columns[3].data[order], np.bincount(inv))
