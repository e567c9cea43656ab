"""Performance cases of the relational operators, through the public API.

Each case is a plain dict of sizes and options.  ``prepare`` makes the inputs
that a program holds before the call (device-resident tables, or a file on
disk for the readers), ``run`` is one pass through the public entry points and
``work`` the bytes that the pass cannot do without: every input column read
once and every output column written once, in the legate layout.

The row order of ``join`` and ``groupby_aggregation`` is unspecified, so their
cases are whole queries, as programs write them: GROUP BY ... ORDER BY the
keys, a join ordered by its event and row ids, or a join with a dimension table
followed by an aggregation per category.  Their outputs are then in a defined
order.

How many rows fall on each key (and which keys match in a join) is the same
for every seed of a case, so that its outputs have the same sizes; the seed
gives the order of the rows, the key values, the strings and all other values.
"""

import os
import sys
import tempfile

import numpy as np
import pyarrow as pa
import pyarrow.csv as pacsv
import pyarrow.parquet as pq
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "legate-dataframe_b200"))

from legate_dataframe import LogicalColumn, LogicalTable  # noqa: E402
from legate_dataframe import _native as N  # noqa: E402
from legate_dataframe.lib.csv import csv_read  # noqa: E402
from legate_dataframe.lib.groupby_aggregation import groupby_aggregation  # noqa: E402
from legate_dataframe.lib.hash_partition import hash_partition  # noqa: E402
from legate_dataframe.lib.join import JoinType, join  # noqa: E402
from legate_dataframe.lib.parquet import parquet_read  # noqa: E402
from legate_dataframe.lib.sort import sort  # noqa: E402

_SHAPE = 20  # seed of the draws that fix how many rows each key has
TS0 = 1_600_000_000_000_000
TS_SPAN = 365 * 86400 * 10**6  # one year in microseconds

# SUM and COUNT (what a dashboard asks of a small table), and the aggregates of
# the 200M-row benchmark: every kind the operator has.
SHORT_AGGS = [("v", "sum", "sum_v"), ("v", "count", "count_v")]
FULL_AGGS = [("v", "sum", "sum_v"), ("v", "mean", "mean_v"), (None, "count_all", "count"),
             ("v", "count", "count_v"), ("i", "min", "min_i"), ("i", "max", "max_i"),
             ("i", "count_distinct", "nunique_i")]


def listed():
    return [
        # The smallest request of the served mix: launches and host time count.
        {"name": "groupby_1k", "op": "groupby", "rows": 1_000, "groups": 100, "zipf": 0.0, "key": "int64",
         "aggs": "short"},
        # The median request of the served mix.
        {"name": "groupby_50k", "op": "groupby", "rows": 50_000, "groups": 5_000, "zipf": 0.0, "key": "int64",
         "aggs": "short"},
        # The benchmark's groupby: skewed keys, float64 with nulls, all aggregates.
        {"name": "groupby_zipf_200m", "op": "groupby", "rows": 200_000_000, "groups": 10_000_000, "zipf": 1.1,
         "key": "int64", "aggs": "full"},
        # Event logs grouped by a string id.
        {"name": "groupby_strings_20m", "op": "groupby", "rows": 20_000_000, "groups": 2_000_000, "zipf": 1.0,
         "key": "string", "aggs": "short"},
        # A join of the served mix: ten rows per key on both sides.
        {"name": "join_inner_50k", "op": "join", "probe": 50_000, "build": 50_000, "dup": 10, "key": "int64",
         "how": "inner"},
        # Two event tables matched on a string id, unmatched rows of both kept.
        {"name": "join_full_strings_1m", "op": "join", "probe": 999_983, "build": 200_003, "dup": 1, "key": "string",
         "how": "full"},
        # The benchmark's join (fact table with a dimension), then an aggregation per category.
        {"name": "join_star_200m", "op": "star", "probe": 200_000_000, "build": 20_000_000, "categories": 10_000},
        # The benchmark's int64 sort: random keys with one int32 column.
        {"name": "sort_int64_100m", "op": "sort", "rows": 100_000_000, "key": "int64"},
        # Event logs ordered by a string id, newest first.
        {"name": "sort_strings_20m", "op": "sort", "rows": 20_000_000, "key": "string_ts"},
        # The local step of a shuffle by a string id.
        {"name": "partition_strings_20m", "op": "partition", "rows": 20_000_000, "key": "string", "parts": 256},
        # Loading an event log from files (in the page cache).
        {"name": "csv_1m", "op": "csv", "rows": 1_000_000},
        {"name": "parquet_4m", "op": "parquet", "rows": 4_000_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case: the same operators over the whole range of sizes."""
    op = rng.choice(["groupby", "groupby", "join", "join", "star", "sort", "sort", "partition", "csv", "parquet"])
    if op == "groupby":
        key = rng.choice(["int64", "int64", "string"])
        rows = _log_int(rng, 1_000, 200_000_000 if key == "int64" else 20_000_000)
        return {"op": op, "rows": rows, "groups": max(2, min(10_000_000, int(rows * rng.choice([0.001, 0.05, 0.1])))),
                "zipf": rng.choice([0.0, 1.0, 1.1]), "key": key, "aggs": rng.choice(["short", "full"])}
    if op == "join":
        key = rng.choice(["int32", "int64", "string"])
        probe = _log_int(rng, 1_000, 1_000_000 if key == "string" else 10_000_000)
        return {"op": op, "probe": probe, "build": max(10, int(probe * rng.choice([0.1, 0.3, 1.0]))),
                "dup": rng.choice([1, 1, 3]), "key": key, "how": rng.choice(["inner", "left", "full"])}
    if op == "star":
        probe = _log_int(rng, 10_000, 200_000_000)
        return {"op": op, "probe": probe, "build": max(10, int(probe * rng.choice([0.01, 0.1]))),
                "categories": rng.choice([25, 1_000, 10_000])}
    if op == "sort":
        key = rng.choice(["int64", "string_ts"])
        return {"op": op, "rows": _log_int(rng, 1_000, 100_000_000 if key == "int64" else 20_000_000), "key": key}
    if op == "partition":
        key = rng.choice(["int64", "string"])
        return {"op": op, "rows": _log_int(rng, 1_000, 20_000_000), "key": key, "parts": rng.choice([2, 8, 64, 256])}
    if op == "csv":
        return {"op": op, "rows": _log_int(rng, 1_000, 1_000_000)}
    return {"op": op, "rows": _log_int(rng, 1_000, 4_000_000)}


# ---- inputs -----------------------------------------------------------------
class _Draws:
    """Seeded draws on the device."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.device)
        self.g.manual_seed(seed)

    def ints(self, lo, hi, n, dtype=torch.int64):
        return torch.randint(lo, hi, (n,), device=self.device, generator=self.g, dtype=dtype)

    def uniform(self, n, dtype=torch.float64):
        return torch.rand(n, device=self.device, generator=self.g, dtype=dtype)

    def normal(self, n, dtype=torch.float64):
        return torch.randn(n, device=self.device, generator=self.g, dtype=dtype)

    def perm(self, n):
        return torch.randperm(n, device=self.device, generator=self.g)

    def ranks(self, n, distinct, s):
        """n draws from [0, distinct): Zipf(s), uniform for s = 0."""
        if s == 0.0:
            return self.ints(0, distinct, n)
        # whole-number weights: their running sums are the same in every run
        weight = torch.arange(1, distinct + 1, device=self.device, dtype=torch.float64).pow(-s) * 2.0**40
        cdf = torch.cumsum(weight.to(torch.int64), 0)
        out = torch.empty(n, dtype=torch.int64, device=self.device)
        for a in range(0, n, 50_000_000):
            b = min(n, a + 50_000_000)
            out[a:b] = torch.searchsorted(cdf, self.ints(0, int(cdf[-1]), b - a), right=True)
        return out

    def shuffled_ranks(self, n, distinct, s):
        """The same n ranks for every seed, in this seed's order."""
        return _Draws(_SHAPE).ranks(n, distinct, s)[self.perm(n)]

    def dictionary(self, n):
        """n strings of 8 to 24 characters [a-z0-9]: [n, 24] bytes (zero-padded) and lengths."""
        lens = _Draws(_SHAPE + 1).ints(8, 25, n)
        abc = torch.tensor(list(b"abcdefghijklmnopqrstuvwxyz0123456789"), dtype=torch.uint8, device=self.device)
        d = abc[self.ints(0, 36, n * 24, dtype=torch.int32).long()].view(n, 24)
        return d * (torch.arange(24, device=self.device) < lens[:, None]), lens


def _string_column(words, lens, pick):
    """Rows words[pick] as a string column."""
    n = pick.numel()
    ln = lens[pick]
    end = torch.cumsum(ln, 0)
    chars = torch.empty(int(end[-1]), dtype=torch.uint8, device=words.device)
    step = 5_000_000
    for a in range(0, n, step):
        b = min(n, a + step)
        w = words[pick[a:b]]
        lo = int(end[a] - ln[a])
        hi = int(end[b - 1])
        chars[lo:hi] = w[torch.arange(24, device=words.device) < ln[a:b, None]]
    ranges = torch.stack([end - ln, end - 1], 1).contiguous()
    return LogicalColumn(pa.string(), N.LDF_STRING, n, ranges.view(torch.uint8).reshape(-1), None, chars=chars,
                         chars_base=0, num_chars=chars.numel())


def _groupby_inputs(case, seed):
    """(key column, key rank of every row, order key of every rank, v, valid, i)."""
    d, n, g = _Draws(seed), case["rows"], case["groups"]
    pick = d.shuffled_ranks(n, g, case["zipf"])
    if case["key"] == "string":
        words, lens = d.dictionary(g)
        key, order = _string_column(words, lens, pick), words
    else:
        order = d.perm(g) * 2_654_435_761 + 12_345
        key = LogicalColumn.from_torch(order[pick], pa.int64())
    v = d.normal(n, torch.float64 if case["key"] == "int64" else torch.float32)
    valid = (d.uniform(n, torch.float32) >= 0.10).to(torch.uint8) if case["key"] == "int64" else None
    i = d.ints(0, 1_000_000, n, torch.int32) if case["aggs"] == "full" else None
    return key, pick, order, v, valid, i


def _prepare_groupby(case, seed):
    key, _, _, v, valid, i = _groupby_inputs(case, seed)
    vt = pa.float64() if v.dtype == torch.float64 else pa.float32()
    cols, names = [key, LogicalColumn.from_torch(v, vt, valid)], ["k", "v"]
    if i is not None:
        cols.append(LogicalColumn.from_torch(i, pa.int32()))
        names.append("i")
    return {"table": LogicalTable(cols, names), "aggs": FULL_AGGS if case["aggs"] == "full" else SHORT_AGGS}


def _join_key(d, kind, ids, space):
    """The key column of rows that hold key id `ids` in [0, space)."""
    if kind == "int32":
        return LogicalColumn.from_torch(ids.to(torch.int32), pa.int32())
    return LogicalColumn.from_torch(ids * 2_654_435_761 + 12_345, pa.int64())


def _prepare_join(case, seed):
    d, n, m, dup = _Draws(seed), case["probe"], case["build"], case["dup"]
    distinct = max(1, m // dup)
    build = torch.arange(m, device=d.device) % distinct
    build = build[d.perm(m)]
    # four probe rows in five hit a build key
    f = _Draws(_SHAPE)
    hit = f.uniform(n, torch.float32) < 0.8
    probe = torch.where(hit, f.ints(0, distinct, n), f.ints(distinct, 2 * distinct, n))[d.perm(n)]
    if case["key"] == "string":
        words, lens = d.dictionary(2 * distinct)
        lk, rk = _string_column(words, lens, probe), _string_column(words, lens, build)
    else:
        lk, rk = _join_key(d, case["key"], probe, 2 * distinct), _join_key(d, case["key"], build, 2 * distinct)
    lhs = LogicalTable([lk, LogicalColumn.from_torch(d.perm(n), pa.int64()),
                        LogicalColumn.from_torch(d.uniform(n), pa.float64())], ["lk", "event", "lv"])
    rhs = LogicalTable([rk, LogicalColumn.from_torch(d.perm(m), pa.int64())], ["rk", "row"])
    return {"lhs": lhs, "rhs": rhs, "how": JoinType[case["how"].upper()]}


def _star_inputs(case, seed):
    """Zipf(0.9) hits on unique int32 build keys, 20% misses, 5% null probe keys."""
    d, n, m = _Draws(seed), case["probe"], case["build"]
    f = _Draws(_SHAPE)
    bkey = d.perm(m).to(torch.int32)
    cat = f.ints(0, case["categories"], m, torch.int32)
    r2 = d.ints(-(2**40), 2**40, m)
    order = d.perm(n)
    rank = f.ranks(n, m, 0.9)[order]
    hit = (f.uniform(n, torch.float32) < 0.8)[order]
    pvalid = (f.uniform(n, torch.float32) >= 0.05)[order]
    pkey = torch.where(hit, bkey[rank], d.ints(m, 2 * m, n, torch.int32))
    return bkey, cat, r2, rank, hit & pvalid, pkey, pvalid, d.uniform(n)


def _prepare_star(case, seed):
    bkey, cat, r2, _, _, pkey, pvalid, lv = _star_inputs(case, seed)
    lhs = LogicalTable([LogicalColumn.from_torch(pkey, pa.int32(), valid=pvalid),
                        LogicalColumn.from_torch(lv, pa.float64())], ["lk", "lv"])
    rhs = LogicalTable([LogicalColumn.from_torch(bkey, pa.int32()), LogicalColumn.from_torch(cat, pa.int32()),
                        LogicalColumn.from_torch(r2, pa.int64())], ["rk", "cat", "r2"])
    return {"lhs": lhs, "rhs": rhs}


def _event_rows(d, n):
    """String ids (Zipf(1.0) over a dictionary a tenth of the rows), timestamps and float32 values."""
    g = max(2, n // 10)
    words, lens = d.dictionary(g)
    key = _string_column(words, lens, d.shuffled_ranks(n, g, 1.0))
    ts = LogicalColumn.from_torch(d.ints(TS0, TS0 + TS_SPAN, n), pa.timestamp("us"))
    return key, ts, LogicalColumn.from_torch(torch.exp(d.normal(n, torch.float32)), pa.float32())


def _prepare_sort(case, seed):
    d, n = _Draws(seed), case["rows"]
    if case["key"] == "string_ts":
        return {"table": LogicalTable(_event_rows(d, n), ["k", "ts", "v"]), "keys": ["k", "ts"],
                "ascending": [True, False]}
    key = d.ints(-(2**62), 2**62, n)
    return {"table": LogicalTable([LogicalColumn.from_torch(key, pa.int64()),
                                   LogicalColumn.from_torch(d.ints(0, 2**30, n, torch.int32), pa.int32())],
                                  ["k", "v"]), "keys": ["k"], "ascending": [True]}


def _prepare_partition(case, seed):
    d, n = _Draws(seed), case["rows"]
    if case["key"] == "string":
        table = LogicalTable(_event_rows(d, n), ["k", "ts", "v"])
    else:
        table = LogicalTable([LogicalColumn.from_torch(d.ints(0, max(2, n // 10), n), pa.int64()),
                              LogicalColumn.from_torch(d.normal(n), pa.float64(),
                                                       d.uniform(n, torch.float32) >= 0.10)], ["k", "v"])
    return {"table": table, "parts": case["parts"]}


def _event_arrow(n, seed):
    """The same rows as a host table: string id, nullable int64, float32."""
    rng, shape = np.random.default_rng(seed), np.random.default_rng(_SHAPE)
    g = max(2, n // 10)
    lens = shape.integers(8, 25, g)
    off = np.zeros(g + 1, np.int32)
    np.cumsum(lens, out=off[1:])
    chars = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz0123456789", np.uint8)[rng.integers(0, 36, int(off[-1]))]
    words = pa.Array.from_buffers(pa.string(), g, [None, pa.py_buffer(off), pa.py_buffer(chars)])
    cdf = np.cumsum(1.0 / np.arange(1, g + 1))
    pick = rng.permutation(np.searchsorted(cdf / cdf[-1], shape.random(n)).clip(max=g - 1))
    count = rng.integers(-(2**40), 2**40, n)
    return pa.table({"k": words.take(pa.array(pick)), "c": pa.array(count, mask=rng.random(n) < 0.1),
                     "v": np.exp(rng.standard_normal(n)).astype(np.float32)})


def _prepare_file(case, seed):
    table = _event_arrow(case["rows"], seed)
    folder = tempfile.TemporaryDirectory()
    path = os.path.join(folder.name, "events." + case["op"])
    if case["op"] == "csv":
        pacsv.write_csv(table, path)
    else:
        pq.write_table(table, path)
    return {"folder": folder, "path": path}


def prepare(case, seed):
    op = case["op"]
    make = {"groupby": _prepare_groupby, "join": _prepare_join, "star": _prepare_star, "sort": _prepare_sort,
            "partition": _prepare_partition, "csv": _prepare_file, "parquet": _prepare_file}[op]
    return {"op": op, **make(case, seed)}


# ---- one pass -----------------------------------------------------------------
_TORCH_OF = {N.LDF_INT32: torch.int32, N.LDF_INT64: torch.int64, N.LDF_TIMESTAMP_US: torch.int64,
             N.LDF_FLOAT32: torch.float32, N.LDF_FLOAT64: torch.float64}


def _columns(table):
    """Every buffer of a table: values (ranges of strings), validity, characters."""
    out = {}
    for name in table.get_column_names():
        c = table.get_column(name)
        if c.ldf_type == N.LDF_STRING:
            out[name] = {"ranges": c.data[: 16 * c.size].view(torch.int64), "chars": c.chars[: c.num_chars]}
        else:
            out[name] = {"data": c.data[: c.size * N.TYPE_WIDTH[c.ldf_type]].view(_TORCH_OF[c.ldf_type])}
        if c.valid is not None:
            out[name]["valid"] = c.valid[: c.size]
    return out


def run(state):
    op = state["op"]
    if op == "groupby":
        return _columns(sort(groupby_aggregation(state["table"], ["k"], state["aggs"]), ["k"]))
    if op == "join":
        t = join(state["lhs"], state["rhs"], lhs_keys=["lk"], rhs_keys=["rk"], join_type=state["how"])
        return _columns(sort(t, ["event", "row"]))
    if op == "star":
        t = join(state["lhs"], state["rhs"], lhs_keys=["lk"], rhs_keys=["rk"], join_type=JoinType.INNER,
                 lhs_out_columns=["lv"], rhs_out_columns=["cat", "r2"])
        t = groupby_aggregation(t, ["cat"], [("lv", "sum", "sum_lv"), ("lv", "mean", "mean_lv"),
                                             ("r2", "sum", "sum_r2"), (None, "count_all", "count")])
        return _columns(sort(t, ["cat"]))
    if op == "sort":
        return _columns(sort(state["table"], state["keys"], sort_ascending=state["ascending"], stable=True))
    if op == "partition":
        table, offsets = hash_partition(state["table"], ["k"], state["parts"])
        return {**_columns(table), "offsets": np.asarray(offsets)}
    if op == "csv":
        return _columns(csv_read(state["path"], dtypes=[pa.string(), pa.int64(), pa.float32()],
                                 names=["k", "c", "v"]))
    return _columns(parquet_read(state["path"]))


# ---- what a pass cannot do without -------------------------------------------
_STRING = 16 + 16  # bytes of a string row: its range and its characters (16 on average)


def _seen(rows, distinct, s):
    """Expected number of distinct values among `rows` draws from Zipf(s)."""
    p = np.arange(1, distinct + 1, dtype=np.float64) ** -s
    return float(-np.expm1(-rows * (p / p.sum())).sum())


def work(case):
    op = case["op"]
    if op == "groupby":
        n, string = case["rows"], case["key"] == "string"
        groups = _seen(n, case["groups"], case["zipf"])
        key, full = _STRING if string else 8, case["aggs"] == "full"
        row = key + (4 if string else 9) + (4 if full else 0)
        return {"bytes": n * row + groups * (key + 17 + (9 + 8 + 4 + 4 + 8 if full else 0)), "flops": 0}
    if op == "join":
        n, m, key = case["probe"], case["build"], {"int32": 4, "int64": 8, "string": _STRING}[case["key"]]
        pairs = 0.8 * n * max(1.0, m / max(1, m // case["dup"]))
        rows = pairs + (0.2 * n if case["how"] != "inner" else 0)
        return {"bytes": n * (key + 16) + m * (key + 8) + rows * (2 * key + 24), "flops": 0}
    if op == "star":
        return {"bytes": case["probe"] * 13 + case["build"] * 16 + case["categories"] * 36, "flops": 0}
    if op == "sort":
        return {"bytes": 2 * case["rows"] * (12 if case["key"] == "int64" else _STRING + 12), "flops": 0}
    if op == "partition":
        return {"bytes": 2 * case["rows"] * (17 if case["key"] == "int64" else _STRING + 12), "flops": 0}
    # the file (about 44 bytes of text a row; Parquet about 14) and the columns
    return {"bytes": case["rows"] * ((44 if op == "csv" else 14) + _STRING + 13), "flops": 0}


# ---- the computed numbers in 64 bits ---------------------------------------------
def _sums(group, v, groups):
    out = torch.zeros(groups, dtype=torch.float64, device=v.device)
    return out.index_add_(0, group, v.double())


def exact(case, seed):
    """Float sums and means per group, in key order; copied columns have none."""
    if case["op"] == "groupby":
        _, pick, order, v, valid, _ = _groupby_inputs(case, seed)
        g = case["groups"]
        if case["key"] == "string":
            words = order.cpu().numpy().view("S24").reshape(-1)
            if len(np.unique(words)) < g:
                return None  # two equal strings in the dictionary
            by_key = torch.from_numpy(np.argsort(words, kind="stable")).to(pick.device)
        else:
            by_key = torch.argsort(order)
        has = torch.ones_like(v, dtype=torch.bool) if valid is None else valid.bool()
        total = _sums(pick, torch.where(has, v, torch.zeros_like(v)), g)
        count = torch.bincount(pick, weights=has.double(), minlength=g)
        used = by_key[torch.bincount(pick, minlength=g)[by_key] > 0]
        out = {"sum_v": {"data": total[used].cpu()}}
        if case["aggs"] == "full":
            out["mean_v"] = {"data": (total[used] / count[used].clamp(min=1)).cpu()}
        return out
    if case["op"] == "star":
        _, cat, _, rank, match, _, _, lv = _star_inputs(case, seed)
        group = cat[rank[match]].long()
        total = _sums(group, lv[match], case["categories"])
        count = torch.bincount(group, minlength=case["categories"])
        used = count > 0
        return {"sum_lv": {"data": total[used].cpu()}, "mean_lv": {"data": (total[used] / count[used]).cpu()}}
    return None
