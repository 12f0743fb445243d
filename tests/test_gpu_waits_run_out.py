"""Kernels that wait for tiles of their own launch, on the B200 with a wait limit of 0 (every wait that is not over
at its first look runs out): a query whose waits ran out never passes an empty or partial result for its own."""
import numpy as np
import pytest
import torch

from vectisdb_b200 import (ColumnCache, ExecuteOptions, GpuEngine, GpuTableRef, make_aggregate, make_column, make_expr,
                           make_filter, make_group_by, make_scan)
from vectisdb_b200.abi import VgpuError
from vectisdb_b200.engine import GpuAggregateKind as A, GpuValueType as T

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


@pytest.mark.parametrize("plan_of", [_select, _groups])
def test_a_result_read_at_once_is_whole_or_an_error(plan_of, table, monkeypatch):
    ref, x, k = table
    monkeypatch.setenv("VGPU_WAIT_LIMIT_NS", "0")
    for _ in range(8):
        r = GpuEngine.instance().execute_plan(plan_of(ref), [], ExecuteOptions(serve_whole_scan_from_cache=True))
        if not r.success:
            assert "in time" in r.error_message, r.error_message
        elif plan_of is _select:
            assert np.array_equal(r.columns[0].data, x[x < 43]) and np.array_equal(r.columns[1].data, k[x < 43])
        else:
            assert np.array_equal(r.columns[0].data, np.unique(k))
            assert np.array_equal(r.columns[2].data, np.bincount(k, minlength=1_000_003)[np.unique(k)])
    torch.cuda.synchronize()
