"""The one-pass row filter's larger tiles for narrow rows on the B200, against numpy: every width around the choice of the
tile, rows around its size, columns that start off a vector's boundary, and predicates over more than the outputs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from vectisdb_b200 import (ExecuteOptions, GpuEngine, device_to_host, make_column, make_expr, make_filter, make_projection,
                           make_scan)
from vectisdb_b200.engine import GpuValueType as T, make_device_column, profile_drain, profile_enable

pytestmark = pytest.mark.gpu
WIDTHS = {1: [T.BOOLEAN], 2: [T.INT16], 4: [T.INT32], 5: [T.INT32, T.BOOLEAN], 8: [T.INT32, T.INT32], 12: [T.INT64, T.INT32],
          13: [T.INT64, T.INT32, T.BOOLEAN]}
NP = {T.BOOLEAN: np.uint8, T.INT16: np.int16, T.INT32: np.int32, T.INT64: np.int64}
C = {T.BOOLEAN: "bool", T.INT16: "short", T.INT32: "int", T.INT64: "long long"}


def _run(plan, cols):
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, cols)
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success, r.error_message
    assert "vgpu_mat_onepass" in names, names
    return [c.data for c in r.columns]


@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("rows", [1, 15, 2047, 2048, 2049, 4097, 300_001])
@pytest.mark.parametrize("width", WIDTHS)
def test_every_width(width, rows, skip):
    rng = np.random.default_rng(rows + width)
    values, cols, keep = [], [], []
    for i, t in enumerate(WIDTHS[width]):
        v = rng.integers(0, 2 if t == T.BOOLEAN else 100, rows + skip).astype(NP[t])
        dev = torch.from_numpy(v).cuda()
        keep.append(dev)
        values.append(v[skip:])
        cols.append(make_device_column(f"c{i}", t, dev.data_ptr() + skip * dev.element_size(), rows))
    torch.cuda.synchronize()
    bound = 1 if WIDTHS[width][0] == T.BOOLEAN else 43
    plan = make_filter([make_expr(f"((bool*)out)[idx] = ((const {C[WIDTHS[width][0]]}*)inputs[0])[row] < {bound};", ["c0"], T.BOOLEAN)],
                       make_scan([c.name for c in cols]))
    got = _run(plan, cols)
    for g, v in zip(got, values):
        assert np.array_equal(g, v[values[0] < bound])


def test_a_narrow_output_of_wide_predicates():
    rng = np.random.default_rng(1)
    n = 100_003
    xs = [rng.standard_normal(n) for _ in range(5)]
    k = rng.integers(0, 1000, n).astype(np.int32)
    cond = " && ".join(f"((const double*)inputs[{i}])[row] < 1.0" for i in range(5))
    names = [f"x{i}" for i in range(5)]
    plan = make_projection([make_expr("((int*)out)[idx] = ((const int*)inputs[0])[row];", ["k"], T.INT32)],
                           make_filter([make_expr(f"((bool*)out)[idx] = {cond};", names, T.BOOLEAN)], make_scan(names + ["k"])))
    got = _run(plan, [make_column(f"x{i}", T.FLOAT64, x) for i, x in enumerate(xs)] + [make_column("k", T.INT32, k)])
    assert np.array_equal(got[0], k[np.all([x < 1.0 for x in xs], axis=0)])


@pytest.mark.parametrize("rows,columns,one_pass", [(1 << 20, 11, True), ((1 << 20) + 1, 11, False), ((1 << 20) + 1, 6, True),
                                                   ((1 << 20) + 1, 7, False)])
def test_wide_rows_of_large_inputs_take_two_passes(rows, columns, one_pass):
    x = (np.arange(rows) % 100).astype(np.int32)
    y = np.arange(rows, dtype=np.int64)
    names = ["x"] + [f"y{i}" for i in range(columns)]
    plan = make_filter([make_expr("((bool*)out)[idx] = ((const int*)inputs[0])[row] < 30;", ["x"], T.BOOLEAN)], make_scan(names))
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, [make_column("x", T.INT32, x)] + [make_column(n, T.INT64, y) for n in names[1:]])
        launched = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    assert r.success and ("vgpu_mat_onepass" in launched) == one_pass, launched
    assert all(np.array_equal(c.data, v[x < 30]) for c, v in zip(r.columns, [x] + [y] * columns))


@pytest.mark.parametrize("bound,estimate,one_pass", [(0, 0, False), (5, 0, False), (60, 0, True), (5, 40_000_000, True)])
def test_a_sample_of_a_large_input_chooses_the_form(bound, estimate, one_pass):
    rows = 46_000_001  # of 12 bytes
    x = (torch.arange(rows, device="cuda") // 7 % 100).to(torch.int32)
    y = torch.arange(rows, device="cuda")
    cols = [make_device_column("x", T.INT32, x.data_ptr(), rows), make_device_column("y", T.INT64, y.data_ptr(), rows)]
    plan = make_filter([make_expr(f"((bool*)out)[idx] = ((const int*)inputs[0])[row] < {bound};", ["x"], T.BOOLEAN)],
                       make_scan(["x", "y"]))
    plan.estimated_rows = estimate
    torch.cuda.synchronize()
    profile_drain()
    profile_enable(True)
    try:
        r = GpuEngine.instance().execute_plan(plan, cols, ExecuteOptions(output_on_device=True))
        names = [rec[0] for rec in profile_drain()]
    finally:
        profile_enable(False)
    got = [device_to_host(c) for c in r.columns]
    r.free()
    assert ("vgpu_mat_onepass" in names) == one_pass and ("vgpu_mat_sample" in names) == (estimate == 0), names
    keep = (x < bound).cpu().numpy()
    assert np.array_equal(got[0], x.cpu().numpy()[keep]) and np.array_equal(got[1], np.flatnonzero(keep))
