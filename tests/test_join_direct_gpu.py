"""Joins at the row counts from which a direct-address table and packed build
records are considered (8,192 build rows under 2^21 probe rows, 131,072 under
fewer): dense integer keys from a negative minimum on, unique and repeated,
against the build row looked up with torch."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["inner", "left"])
@pytest.mark.parametrize("width", [16, 32, 64])
@pytest.mark.parametrize("m, n", [(8191, 1 << 21), (8192, (1 << 21) - 1), (8192, 1 << 21), (32000, (1 << 21) + 3),
                                  (131071, 1 << 21), (131072, 5000)])
def test_dense_keys(m, n, width, how):
    import pyarrow as pa
    import torch

    from legate_dataframe import LogicalColumn, LogicalTable
    from legate_dataframe.lib.join import JoinType, join

    if width == 16 and m > 32000:
        pytest.skip("more keys than int16 has")
    dt, at = {16: (torch.int16, pa.int16()), 32: (torch.int32, pa.int32()), 64: (torch.int64, pa.int64())}[width]
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n)
    lowest = -500
    for repeats in (0, 1):
        b = torch.randperm(m, device="cuda", generator=g)
        p = torch.randint(-100, m + 100, (n,), device="cuda", generator=g)
        if repeats:
            b[0] = b[1]  # one key twice, one not at all
        pay = torch.randint(-2**40, 2**40, (2, m), device="cuda", generator=g)
        lhs = LogicalTable([LogicalColumn.from_torch((p + lowest).to(dt), at),
                            LogicalColumn.from_torch(torch.arange(n, device="cuda"), pa.int64())], ["k", "a"])
        rhs = LogicalTable([LogicalColumn.from_torch((b + lowest).to(dt), at),
                            LogicalColumn.from_torch(pay[0], pa.int64()),
                            LogicalColumn.from_torch(pay[1].to(torch.int32), pa.int32())], ["r", "b", "c"])
        out = join(lhs, rhs, lhs_keys=["k"], rhs_keys=["r"], join_type=JoinType[how.upper()])
        order = torch.argsort(b, stable=True)
        first = torch.searchsorted(b[order], p)
        many = torch.searchsorted(b[order], p, right=True) - first
        rows = many if how == "inner" else many.clamp(min=1)
        assert out.num_rows() == int(rows.sum())

        def column(name, t):
            c = out.get_column(name)
            return c.data[: c.size * t.itemsize].view(t)

        a = column("a", torch.int64)
        assert bool((torch.bincount(a, minlength=n) == rows).all())
        assert bool((column("k", dt).long() - lowest == p[a]).all())
        hit = many[a] > 0
        if how == "left":
            for name in ("r", "b", "c"):
                c = out.get_column(name)
                assert bool((c.valid[: c.size].bool() == hit).all())
        got_b, got_c, got_r = column("b", torch.int64)[hit], column("c", torch.int32)[hit], column("r", dt)[hit]
        assert bool((got_r.long() - lowest == p[a][hit]).all())
        # the build row of each output row: its payload tells, and each of a key's rows comes once per probe row
        lookup = torch.sort(pay[0])
        at_row = lookup.indices[torch.searchsorted(lookup.values, got_b).clamp(max=m - 1)]
        assert bool((pay[0][at_row] == got_b).all()) and bool((pay[1][at_row].to(torch.int32) == got_c).all())
        assert bool((b[at_row] == p[a][hit]).all())
        pairs = a[hit] * m + at_row
        assert pairs.unique().numel() == pairs.numel()
