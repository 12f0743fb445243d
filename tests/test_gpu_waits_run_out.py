"""Kernels that wait for tiles of their own launch, on the B200 with a wait limit of 0 (every wait that is not over
at its first look runs out): a query whose waits ran out never passes an empty or partial result for its own; where the
result is read at once, another form gives it."""
import numpy as np
import pytest
import torch

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, device_to_host, make_aggregate, make_column,
                           make_expr, make_filter, make_group_by, make_join, make_scan)
from vectisdb_b200.abi import VgpuError
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
N = 3_000_017


@pytest.fixture
def table():
    ref = GpuTableRef("memory", "main", "waits")
    x = (np.arange(N) % 100).astype(np.int32)
    k = ((np.arange(N) * 7919) % 1_000_003).astype(np.int32)
    ColumnCache.put_table(ref, [make_column("x", T.INT32, x), make_column("k", T.INT32, k)])
    yield ref, x, k
    ColumnCache.invalidate_table(ref)


def _select(ref):
    return make_filter([make_expr("((bool*)out)[idx] = (((const int*)inputs[0])[row] < 43);", ["x"], T.BOOLEAN)],
                       make_scan(["x", "k"], ref))


def _groups(ref):
    return make_group_by(["k"], [make_aggregate(A.SUM, "x", T.HUGEINT), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["x", "k"], ref))


@pytest.mark.parametrize("plan_of", [_select, _groups])
def test_a_count_left_on_the_device_says_so_when_it_is_read(plan_of, table, monkeypatch):
    ref, _, _ = table
    monkeypatch.setenv("VGPU_WAIT_LIMIT_NS", "0")
    lazy = ExecuteOptions(serve_whole_scan_from_cache=True, output_on_device=True, no_sync=True,
                          stream=torch.cuda.Stream().cuda_stream)
    for _ in range(8):
        r = GpuEngine.instance().execute_plan(plan_of(ref), [], lazy)
        with pytest.raises(VgpuError, match="not completed on the device"):
            r.columns
        r.free()
    torch.cuda.synchronize()  # the context is in order


@pytest.mark.parametrize("plan_of,general", [(_select, "vgpu_mat_count"), (_groups, "vgpu_gb_part_count")])
@pytest.mark.parametrize("on_device", [False, True])
def test_a_result_read_at_once_takes_the_general_form(plan_of, general, on_device, table, monkeypatch):
    ref, x, k = table
    monkeypatch.setenv("VGPU_WAIT_LIMIT_NS", "0")
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan_of(ref), [], ExecuteOptions(serve_whole_scan_from_cache=True,
                                                                               output_on_device=on_device))
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    if not on_device:
        assert r.success, r.error_message
    got = [device_to_host(c) if on_device else c.data for c in r.columns]
    if on_device:
        r.free()
    assert general in names and ("vgpu_mat_onepass" in names or "vgpu_gb_l2" in names), names
    if plan_of is _select:
        assert np.array_equal(got[0], x[x < 43]) and np.array_equal(got[1], k[x < 43])
    else:
        order = np.argsort(got[0])
        assert np.array_equal(got[0][order], np.unique(k))
        assert np.array_equal(got[2][order], np.bincount(k, minlength=1_000_003)[np.unique(k)])


def test_a_join_whose_count_ran_out_is_expanded(monkeypatch):
    rng = np.random.default_rng(1)
    rk, lk = rng.permutation(300_000).astype(np.int64), rng.integers(0, 300_000, 500_000).astype(np.int64)
    plan = make_join("lk", "rk", ["lk", "b"], make_scan(["lk"]), make_scan(["rk", "b"]))
    monkeypatch.setenv("VGPU_WAIT_LIMIT_NS", "0")
    r = GpuEngine.instance().execute_plan(plan, [make_column("lk", T.INT64, lk), make_column("rk", T.INT64, rk),
                                                 make_column("b", T.INT64, rk * 3)])
    assert r.success, r.error_message
    assert np.array_equal(r.columns[0].data, lk) and np.array_equal(r.columns[1].data, lk * 3)
