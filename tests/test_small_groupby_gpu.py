"""Groupby of small inputs (one cluster kernel) at the edges of its warps,
clusters and row limit, against the oracle."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from oracle import relational as R

pytestmark = pytest.mark.gpu

AGGS = [("f", "sum", "sum_f"), ("f", "mean", "mean_f"), ("f", "min", "min_f"), ("i", "sum", "sum_i"),
        ("i", "max", "max_i"), ("i", "min", "min_i"), ("i", "count", "count_i"), (None, "count_all", "rows"),
        ("c", "count_distinct", "nd_c"), ("l", "count_distinct", "nd_l"), ("l", "max", "max_l")]


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 8192, 65537, 131072, 131073])
@pytest.mark.parametrize("key", ["i64", "i8", "str", "pair"])
@pytest.mark.parametrize("groups", [1, 300, None])
def test_small_groupby(n, key, groups):
    """Every aggregate over one group, groups around the shared-memory
    records' limit and one group per row; null keys, the key words that mark
    an empty slot in either plan; tolerance: sums are exact fixed point
    rounded once, the oracle's are compensated, so they agree to a few ulps."""
    rng = np.random.default_rng(n)
    g = rng.integers(0, groups, n) if groups else rng.permutation(n)
    i64 = g.astype(np.int64) * 2_654_435_761
    i64[g == 0] = -1
    i64[g == 1] = 0x7FF4DEAD7FF4BEEF
    knull = (g % 7 == 3) if groups != 1 else None
    cols = {"i64": ["k"], "i8": ["k8"], "str": ["ks"], "pair": ["k", "k8"]}[key]
    t = pa.table({"k": pa.array(i64, mask=knull), "k8": pa.array((g % 256).astype(np.uint8).view(np.int8), mask=knull),
                  "ks": pa.array([f"key {x * 7919 % 100003}{'y' * (x % 40)}" for x in g.tolist()], mask=knull),
                  "f": pa.array(rng.normal(size=n), mask=rng.random(n) < 0.2),
                  "i": pa.array(rng.integers(-2**31, 2**31, n).astype(np.int32), mask=rng.random(n) < 0.1),
                  "c": rng.integers(0, 50, n).astype(np.int16),
                  "l": pa.array(rng.integers(-2**40, 2**40, n) // 2**36)})
    from legate_dataframe import LogicalTable
    from legate_dataframe.lib.groupby_aggregation import groupby_aggregation

    res = groupby_aggregation(LogicalTable.from_arrow(t), cols, AGGS).to_arrow()
    assert_tables_equal(res, R.groupby(t, cols, AGGS), sort_by=cols, rtol=1e-12)
