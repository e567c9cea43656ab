"""Sorts of small tables (one counting kernel instead of radix passes) at the
edges of its blocks, tiles and row limit, against the oracle."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from oracle import relational as R
from test_sort_gpu import run_sort

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 1023, 1025, 2048, 2049, 16383, 16384, 16385]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("keys", [["i"], ["f", "i"], ["b", "f", "g"], ["i", "f", "g", "u"]])
def test_small_sort_keys(n, keys):
    """One to three words of key, classes of nulls and NaNs, ties, both
    directions and null placements, a limit from either end; the last key
    list is wider than three words and takes the radix passes."""
    rng = np.random.default_rng(n)
    f = rng.integers(-20, 20, n).astype(np.float64)
    f[::7] = np.nan
    f[::11] = -0.0
    f[::13] = np.inf
    t = pa.table({"i": rng.integers(-2**63, 2**63 - 1, n) >> rng.integers(0, 64, n),
                  "f": pa.array(f, mask=rng.random(n) < 0.2),
                  "b": rng.random(n) < 0.5,
                  "g": pa.array(rng.integers(-3, 3, n), pa.int64(), mask=rng.random(n) < 0.2),
                  "u": rng.integers(0, 2**16, n).astype(np.uint16),
                  "s": [f"r{i}" for i in range(n)], "row": np.arange(n)})
    asc = [bool(j % 2) for j in range(len(keys))]
    for nulls_at_end, limit in ((True, None), (False, max(1, n // 3)), (True, -max(1, n // 2))):
        res = run_sort(t, keys, asc, nulls_at_end, limit=limit)
        exp = R.sort(t, keys, asc, nulls_at_end, limit=limit)
        assert res.column("row").equals(exp.column("row"))
        assert_tables_equal(res, exp, sort_by=None)


@pytest.mark.parametrize("n", [33, 5000, 16384, 30000])
def test_small_string_ranks(n):
    """Few distinct strings: equal 32-byte heads with different tails and
    lengths, prefixes, zero bytes, nulls; more rows than the small sort takes."""
    rng = np.random.default_rng(n)
    head = "h" * 32
    words = ["", "a", "a\x00", "a\x00\x00", "ab", head, head + "\x00", head + "a", head + "ab", head + "b",
             head[:31], "\U0001F642", "\x7f"] + [f"{head[:i % 33]}{i}" for i in range(4000)]
    s = pa.array([words[i] for i in rng.integers(0, len(words), n)], mask=rng.random(n) < 0.05)
    t = pa.table({"s": s, "v": rng.integers(0, 4, n), "row": np.arange(n)})
    for asc, nulls_at_end in (([True, True], True), ([False, True], False)):
        res = run_sort(t, ["s", "v"], asc, nulls_at_end)
        assert_tables_equal(res, R.sort(t, ["s", "v"], asc, nulls_at_end), sort_by=None)
