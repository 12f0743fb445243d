"""GROUP BY keys that pack into 60 to 63 bits on the B200: such a key space times the state words per
slot exceeds 2^64 bytes, and the query runs by hashed partitioning like any other sparse key."""
import numpy as np
import pytest

from vectisdb_b200 import GpuEngine, make_aggregate, make_column, make_group_by, make_scan
from vectisdb_b200.engine import GpuAggregateKind as A, GpuTableRef, GpuValueType as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [59, 60, 61, 63])
def test_sum_and_count_by_a_key_of_up_to_63_bits(bits):
    rng = np.random.default_rng(bits)
    n = 50_003
    ids = rng.integers(0, 1 << bits, 2000, dtype=np.int64)
    ids[:2] = [0, (1 << bits) - 1]  # the packed key uses every bit
    k = ids[rng.integers(0, len(ids), n)]
    k[:2] = ids[:2]
    v = rng.integers(-(1 << 40), 1 << 40, n).astype(np.float64)  # whole numbers: every order of adding is exact
    plan = make_group_by(["k"], [make_aggregate(A.SUM, "v", T.FLOAT64), make_aggregate(A.COUNT_STAR, "", T.INT64)],
                         make_scan(["k", "v"], GpuTableRef("memory", "main", "wide")))
    r = GpuEngine.instance().execute_plan(plan, [make_column("k", T.INT64, k), make_column("v", T.FLOAT64, v)])
    assert r.success, r.error_message
    keys, inv, counts = np.unique(k, return_inverse=True, return_counts=True)
    order = np.argsort(r.columns[0].data)
    assert np.array_equal(r.columns[0].data[order], keys)
    assert np.array_equal(r.columns[1].data[order], np.bincount(inv, weights=v))
    assert np.array_equal(r.columns[2].data[order], counts)
