"""Groupbys of up to 131,072 rows with several NUNIQUE columns on either side of the
line up to which the small plan takes them, against the oracle; the plan is told
from the kernels that ran."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from oracle import relational as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, columns, small", [(131072, 4, True), (131072, 5, False), (104857, 5, True), (104858, 5, False),
                                               (87381, 6, True), (87382, 6, False), (131072, 0, True)])
def test_line_between_the_plans(n, columns, small):
    from legate_dataframe import LogicalTable
    from legate_dataframe import _native as N
    from legate_dataframe.lib.groupby_aggregation import groupby_aggregation

    rng = np.random.default_rng(columns)
    cols = {f"c{i}": pa.array(rng.integers(0, 40 * (i + 1), n), mask=rng.random(n) < 0.1) for i in range(6)}
    t = pa.table({"k": rng.integers(0, 3000, n) * 7919, **cols})
    aggs = [(f"c{i}", "count_distinct", f"n{i}") for i in range(columns)] + [(f"c{i}", "sum", f"s{i}") for i in range(6)]
    lt = LogicalTable.from_arrow(t)
    N.profile_enable(True)
    N.profile_report(reset=True)
    try:
        res = groupby_aggregation(lt, ["k"], aggs)
        kernels = N.profile_report(reset=True)
    finally:
        N.profile_enable(False)
    assert ("small_groupby" in kernels) == small
    assert_tables_equal(res.to_arrow(), R.groupby(t, ["k"], aggs), sort_by=["k"])
