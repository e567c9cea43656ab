"""Joins whose build keys repeat (rows listed per slot, output rows shared out
over a tile's threads) at the edges of probe tiles and of the direct-address
table's row limit, against the oracle."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from oracle import relational as R
from test_join_gpu import HOW

pytestmark = pytest.mark.gpu


def run_join(lhs, rhs, keys, how, nulls_equal):
    from legate_dataframe import LogicalTable
    from legate_dataframe.lib.join import join

    out_r = [] if how in ("semi", "anti") else None
    return join(LogicalTable.from_arrow(lhs), LogicalTable.from_arrow(rhs), lhs_keys=keys,
                rhs_keys=["r" + k for k in keys], join_type=HOW[how], nulls_equal=nulls_equal,
                rhs_out_columns=out_r).to_arrow()


def tables(n, m, kind, seed):
    """Build keys of 1 to some 40 rows, one key of m // 8 rows that a few probe
    rows hit, null keys on both sides, the key word that marks an empty slot."""
    rng = np.random.default_rng(seed)
    space = max(2, m // 10)
    b, p = rng.integers(0, space, m), rng.integers(0, 2 * space, n)
    b[: m // 8] = 1
    p[p == 1] = 2
    p[:3] = 1
    rng.shuffle(b)
    bn, pn = rng.random(m) < min(0.02, 50 / m), rng.random(n) < min(0.02, 50 / n)
    if kind == "dense":
        bk, pk = b.astype(np.int32), p.astype(np.int32)
    elif kind == "int64":
        bk, pk = b * 2_654_435_761 - 2_654_435_762, p * 2_654_435_761 - 2_654_435_762  # key id 1 is -1
    else:
        bk, pk = [f"key{x * 7919 % 100003}" for x in b], [f"key{x * 7919 % 100003}" for x in p]
    lhs = {"k": pa.array(pk, mask=pn), "a": np.arange(n), "s": [f"l{i % 97}" for i in range(n)]}
    rhs = {"rk": pa.array(bk, mask=bn), "b": np.arange(m).astype(np.int32), "c": pa.array(rng.normal(size=m))}
    keys = ["k"]
    if kind == "pair":
        lhs["q"], rhs["rq"] = pa.array(p % 3, mask=pn), pa.array(b % 3, mask=bn)
        keys = ["k", "q"]
    return pa.table(lhs), pa.table(rhs), keys


@pytest.mark.parametrize("how", list(HOW))
@pytest.mark.parametrize("nulls_equal", [True, False])
@pytest.mark.parametrize("kind", ["dense", "int64", "string", "pair"])
@pytest.mark.parametrize("n, m", [(1, 16), (1023, 300), (1025, 3000), (5000, 1024)])
def test_join_repeated_keys(n, m, kind, nulls_equal, how):
    lhs, rhs, keys = tables(n, m, kind, n + m)
    res = run_join(lhs, rhs, keys, how, nulls_equal)
    exp = R.join(lhs, rhs, keys, ["r" + k for k in keys], how, nulls_equal)
    by = [c for c in ("a", "b") if c in exp.column_names]
    assert_tables_equal(res, exp, sort_by=by)


@pytest.mark.parametrize("how", ["inner", "full", "semi"])
@pytest.mark.parametrize("kind", ["dense", "int64"])
@pytest.mark.parametrize("m", [131071, 131072])
def test_join_repeated_keys_large_build(m, kind, how):
    lhs, rhs, keys = tables(2049, m, kind, m)
    res = run_join(lhs, rhs, keys, how, True)
    by = ["a"] if how == "semi" else ["a", "b"]
    assert_tables_equal(res, R.join(lhs, rhs, keys, ["rk"], how, True), sort_by=by)
