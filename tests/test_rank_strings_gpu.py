"""Ranks of up to 8,192 distinct strings that share long prefixes: rounds of 32
and then 24 bytes at their edges, strings that end in NULs or are prefixes of one
another, against Python's order of their bytes."""

import numpy as np
import pyarrow as pa
import pytest

from test_sort_gpu import run_sort

pytestmark = pytest.mark.gpu


def check(strings):
    rows = np.random.default_rng(len(strings)).integers(0, len(strings), 2 * len(strings))
    data = [strings[i] for i in rows]
    t = pa.table({"k": pa.array(data, pa.string()), "row": np.arange(len(data))})
    got = run_sort(t, ["k"], [True]).column("row").to_numpy()
    assert np.array_equal(got, sorted(range(len(data)), key=lambda i: (data[i].encode(), i)))


@pytest.mark.parametrize("prefix", [0, 31, 32, 33, 55, 56, 57, 80, 500])
@pytest.mark.parametrize("n", [40, 4000])
def test_common_prefix(prefix, n):
    rng = np.random.default_rng(prefix)
    tails = {"".join(map(chr, rng.integers(97, 100, rng.integers(0, 12)))) for _ in range(n)}
    check(["p" * prefix + t for t in tails])


def test_prefixes_of_one_another_and_trailing_nuls():
    base = "ab" * 100
    check(sorted({base[:k] + z for k in range(len(base)) for z in ("", "\0", "\0\0", "\0x", "\x01")}))


def test_a_few_rounds_behind_different_prefixes():
    rng = np.random.default_rng(3)
    check(sorted({p + "x" * int(k) + t for p in ("", "q" * 30, "q" * 60, "r" * 90)
                  for k in rng.integers(0, 200, 300) for t in ("", "1", "22")}))


def test_rounds_are_no_more_than_the_strings_need():
    """Launches, not time: strings of 400 bytes that differ at once take one
    round, those behind a common prefix of 200 bytes one for 32 and eight of 24."""
    from legate_dataframe import LogicalTable
    from legate_dataframe import _native as N
    from legate_dataframe.lib.sort import sort

    def rounds(strings):
        t = LogicalTable.from_arrow(pa.table({"k": strings}))
        N.profile_enable(True)
        N.profile_report(reset=True)
        try:
            sort(t, ["k"])
            return N.profile_report(reset=True)["rank_strings"][0]
        finally:
            N.profile_enable(False)

    rng = np.random.default_rng(4)
    ids = [f"{i:05d}" for i in rng.permutation(3000)]
    assert rounds(ids) == 1
    assert rounds([i + "x" * 395 for i in ids]) == 1
    assert rounds(["p" * 200 + i for i in ids]) == 9
