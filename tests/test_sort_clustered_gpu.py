"""Sorts of 2^21 rows and more whose equal keys stand in neighbouring rows, as in
event logs: the sampled rows must show such groups whatever their length, so
that no long runs of equal words are left to order row against row.  Groups that
the sample does not see are ordered by a thread, by a block, or, over 4,096
rows, by sorting the whole word."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from test_sort_gpu import run_sort

pytestmark = pytest.mark.gpu

N = (1 << 21) + 5
SAMPLE = 1 << 17


def sampled_rows(n):
    """sample_row of legate-dataframe_b200/csrc/radix.cu."""
    bits = int(n - 1).bit_length()
    x = np.arange(SAMPLE, dtype=np.uint64)
    out = np.zeros(SAMPLE, bool)
    while not out.all():
        y = x.copy()
        for _ in range(3):
            y = ((y * np.uint64(0x9E3779B1) + np.uint64(0x85EBCA6B)) & np.uint64(0xFFFFFFFF)) & np.uint64(2**bits - 1)
            y ^= y >> np.uint64((bits + 1) // 2)
        x = np.where(out, x, y)
        out |= x < n
    assert len(np.unique(x)) == SAMPLE
    return x.astype(np.int64)


def beside(n, kind):
    cols = {"a": np.arange(n, dtype=np.int32)}
    if kind == "wide":  # over 8 bytes: row ids
        cols["b"] = np.arange(n)
    return cols


def check(key, kind, asc=True):
    t = pa.table({"k": key, **beside(len(key), kind)})
    order = np.argsort(key if asc else ~key, kind="stable")
    assert_tables_equal(run_sort(t, ["k"], [asc]), t.take(pa.array(order)), sort_by=None)


@pytest.mark.parametrize("kind", ["pair", "wide"])
@pytest.mark.parametrize("cluster", [33, 3000, 4096, 4097, 9000])
def test_groups_that_no_sampled_row_shows(cluster, kind):
    rng = np.random.default_rng(cluster)
    v = rng.integers(-2**62, 2**62, N)
    seen = np.zeros(N, bool)
    seen[sampled_rows(N)] = True
    at = np.flatnonzero(~seen)[:: N // 20_000][:cluster]
    assert len(at) == cluster
    v[at] = (v[5] & ~np.int64(0xFFFF)) | rng.integers(0, 1 << 16, cluster)
    v[at[::2]] = v[5]
    check(v, kind, cluster % 2 == 0)


@pytest.mark.parametrize("kind", ["pair", "wide"])
@pytest.mark.parametrize("group", [2, 16, 40, 700, 5000])
def test_neighbouring_equal_keys(group, kind):
    rng = np.random.default_rng(group)
    check(rng.integers(-2**62, 2**62, N // group + 1).repeat(group)[:N], kind)
    check(np.sort(rng.integers(-2**62, 2**62, N // group + 1)).repeat(group)[:N], kind, asc=False)


@pytest.mark.parametrize("kind", ["pair", "wide"])
def test_groups_shorter_than_the_sample_stride_are_seen(kind):
    """20M rows in groups of 100, one row in 153 sampled: no run of equal words
    is listed for a block to order."""
    import torch

    from legate_dataframe import LogicalColumn, LogicalTable
    from legate_dataframe import _native as N_
    from legate_dataframe.lib.sort import sort

    n = 20_000_000
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    key = torch.randint(-2**62, 2**62, (n // 100,), device="cuda", generator=g).repeat_interleave(100)
    cols = [LogicalColumn.from_torch(key, pa.int64()),
            LogicalColumn.from_torch(torch.arange(n, device="cuda", dtype=torch.int32), pa.int32())]
    names = ["k", "row"]
    if kind == "wide":
        cols.append(LogicalColumn.from_torch(key, pa.int64()))
        names.append("b")
    N_.profile_enable(True)
    N_.profile_report(reset=True)
    try:
        out = sort(LogicalTable(cols, names), ["k"])
        torch.cuda.synchronize()
        kernels = N_.profile_report(reset=True)
    finally:
        N_.profile_enable(False)
    assert "order_pair_runs" not in kernels and "order_runs" not in kernels
    k = out.get_column("k").data[: 8 * n].view(torch.int64)
    row = out.get_column("row").data[: 4 * n].view(torch.int32).long()
    assert bool((k == key[row]).all()) and bool((k[1:] >= k[:-1]).all())
    assert bool(((k[1:] > k[:-1]) | (row[1:] > row[:-1])).all())
