"""Joins whose build side has few repeated keys: the rows marked as repeats (one
bit each) at the edges of the marks' words, repeats of a null key and of the key
word that marks an empty slot, against the oracle; and the cost of listing them,
which must follow the repeats and not the build rows."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from oracle import relational as R
from test_join_repeats_gpu import run_join

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["inner", "left", "full"])
@pytest.mark.parametrize("kind", ["int32", "int64", "string", "pair"])
@pytest.mark.parametrize("m", [2, 31, 32, 33, 64, 65, 257, 131073])
def test_marked_rows(m, kind, how):
    rng = np.random.default_rng(m)
    b = rng.permutation(m).astype(np.int64) - 1  # -1: the empty slot's word
    b[-1] = b[0]
    b[m // 2] = -1
    nulls = np.zeros(m, bool)
    nulls[[0, m - 1]] = m > 40
    n = 1500
    p = rng.integers(-1, m + m // 4 + 1, n)
    pn = rng.random(n) < min(0.05, 20 / n)

    def column(x, mask):
        if kind == "string":
            return pa.array([f"k{v}" for v in x.tolist()], mask=mask)
        return pa.array(x.astype(np.int32) if kind == "int32" else x, mask=mask)

    lhs, rhs, keys = {"k": column(p, pn), "a": np.arange(n)}, {"rk": column(b, nulls), "b": np.arange(m)}, ["k"]
    if kind == "pair":
        lhs["q"], rhs["rq"], keys = pa.array(p % 2, mask=pn), pa.array(b % 2, mask=nulls), ["k", "q"]
    lhs, rhs = pa.table(lhs), pa.table(rhs)
    for nulls_equal in (True, False):
        res = run_join(lhs, rhs, keys, how, nulls_equal)
        exp = R.join(lhs, rhs, keys, ["r" + k for k in keys], how, nulls_equal)
        assert_tables_equal(res, exp, sort_by=["a", "b"])


@pytest.mark.parametrize("dense", [True, False])
def test_listing_follows_the_repeats(dense):
    """20M build rows with 1 % repeats: device time of listing them against the
    build's (listing every row took as long again or longer)."""
    import torch

    from legate_dataframe import LogicalColumn, LogicalTable
    from legate_dataframe import _native as N
    from legate_dataframe.lib.join import JoinType, join

    m, n = 20_000_000, 1_000_000
    b = torch.randperm(m, device="cuda")
    b[: m // 100] = b[m // 100: 2 * (m // 100)]
    b = b[torch.randperm(m, device="cuda")]
    p = torch.randint(0, m, (n,), device="cuda")
    if dense:
        b, p, t = b.int(), p.int(), pa.int32()
    else:
        b, p, t = b * 2_654_435_761, p * 2_654_435_761, pa.int64()
    lhs = LogicalTable([LogicalColumn.from_torch(p, t)], ["k"])
    rhs = LogicalTable([LogicalColumn.from_torch(b, t)], ["r"])
    kernels = {}
    for profiled in (False, True):  # the first call warms up
        N.profile_enable(profiled)
        N.profile_report(reset=True)
        try:
            res = join(lhs, rhs, lhs_keys=["k"], rhs_keys=["r"], join_type=JoinType.INNER)
            torch.cuda.synchronize()
            kernels = N.profile_report(reset=True)
        finally:
            N.profile_enable(False)
    repeats = torch.zeros(m, dtype=torch.int64, device="cuda").scatter_add_(
        0, (b.long() if dense else b // 2_654_435_761), torch.ones(m, dtype=torch.int64, device="cuda"))
    assert res.num_rows() == int(repeats[p.long() if dense else p // 2_654_435_761].sum())
    build = kernels["direct_build" if dense else "build"][1]
    assert kernels["csr_count"][1] + kernels["csr_fill"][1] < 0.5 * build, kernels
