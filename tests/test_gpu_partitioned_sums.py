"""Integer sums of the direct-partitioned group-by on either side of 64 bits, on the B200, against exact integers:
with and without pre-aggregated heavy keys (warp-combined or row by row), with split partitions, and keys of 64-bit
columns far from zero, whose packed form takes 32 bits."""
import numpy as np
import pytest

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column,
                           make_group_by, make_scan)
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, hugeint_to_int, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
N = 300_007
LIMITS = [1 << 20, ((1 << 63) - 1) // N, ((1 << 63) - 1) // N + 1, 1 << 62]


@pytest.mark.parametrize("env", [{"VGPU_GB_HEAVY": "0"}, {"VGPU_GB_HEAVY": "0", "VGPU_GB_BUCKET_PLAIN": "1"},
                                 {"VGPU_GB_HEAVY": "0", "VGPU_GB_SPLIT_ROWS": "256"},
                                 {"VGPU_GB_HEAVY": "0", "VGPU_GB_DIRECT_BITS": "13"}, {"VGPU_GB_HEAVY": "2"},
                                 {"VGPU_GB_HEAVY": "2", "VGPU_GB_DIRECT_BITS": "13"},
                                 {"VGPU_GB_HEAVY": "2", "VGPU_GB_HEAVY_WARP": "0"},
                                 {"VGPU_GB_HEAVY": "2", "VGPU_GB_STAGED": "0", "VGPU_GB_SPLIT_ROWS": "256"}])
@pytest.mark.parametrize("limit", LIMITS)
def test_cached_integer_sums_on_either_side_of_64_bits(limit, env, monkeypatch):
    monkeypatch.setenv("VGPU_GB_STRATEGY", "direct")
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    rng = np.random.default_rng(4)
    base = -(1 << 61) + 12_345
    k = rng.integers(0, 50_000, N)
    k[: N // 2] = 49_999  # half the rows, all of the largest value, on one key
    v = rng.integers(-limit, limit, N, dtype=np.int64, endpoint=True)
    v[: N // 2], v[-1] = limit, -limit
    w = rng.integers(-(1 << 15), 1 << 15, N).astype(np.int16)
    order = rng.permutation(N)
    k, v, w = k[order] + base, v[order], w[order]
    ref = GpuTableRef("memory", "main", "psums")
    cols = [make_column("k", T.INT64, k), make_column("v", T.INT64, v), make_column("w", T.INT16, w)]
    # heavy keys take 8-byte value columns only
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.HUGEINT), make_aggregate(A.COUNT_STAR, "", T.INT64)] +
                         ([] if env["VGPU_GB_HEAVY"] == "2" else [make_aggregate(A.SUM, "w", T.HUGEINT)]),
                         make_scan(["k", "v", "w"], ref))
    ColumnCache.put_table(ref, cols)
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [], ExecuteOptions(serve_whole_scan_from_cache=True))
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
        ColumnCache.invalidate_table(ref)
    assert r.success, r.error_message
    assert "vgpu_gb_dbucket" in names and ("heavy_select" in names) == (env["VGPU_GB_HEAVY"] == "2"), names
    exp = {}
    for key, x, y in zip(k.tolist(), v.tolist(), w.tolist()):
        s, t, c = exp.get(key, (0, 0, 0))
        exp[key] = (s + x, t + y, c + 1)
    sums, counts = hugeint_to_int(r.columns[1].data), r.columns[2].data.tolist()
    small = hugeint_to_int(r.columns[3].data) if len(r.columns) > 3 else [exp[key][1] for key in r.columns[0].data.tolist()]
    assert dict(zip(r.columns[0].data.tolist(), zip(sums, small, counts))) == exp
