"""Whole-table sorts of 2^21 rows and more whose rows travel through the passes
(one integer key, at most 8 bytes beside it), and the same keys with columns
that do not fit, against numpy's stable sort."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from test_sort_gpu import run_sort
from test_sort_leading_bits_gpu import N, STRIDE, none, stable_order

pytestmark = pytest.mark.gpu

BESIDE = {
    "i32": lambda r, n: {"a": np.arange(n, dtype=np.int32)},
    "i64": lambda r, n: {"a": r.integers(-2**63, 2**63 - 1, n)},
    "f64": lambda r, n: {"a": np.where(r.random(n) < 0.1, np.nan, r.normal(size=n))},
    "i8": lambda r, n: {"a": r.integers(-128, 128, n).astype(np.int8)},
    "packed4": lambda r, n: {"a": r.random(n) < 0.5, "b": r.integers(0, 2**16, n).astype(np.uint16)},
    "packed8": lambda r, n: {"a": r.integers(-9, 9, n).astype(np.int8), "b": r.normal(size=n).astype(np.float32),
                             "c": r.integers(-2**15, 2**15, n).astype(np.int16), "d": r.random(n) < 0.5},
    "i32i32": lambda r, n: {"a": np.arange(n, dtype=np.int32), "b": r.integers(-2**31, 2**31, n).astype(np.int32)},
    "wide": lambda r, n: {"a": np.arange(n), "b": r.integers(0, 9, n).astype(np.int8)},  # 9 bytes: row ids
    "null": lambda r, n: {"a": pa.array(np.arange(n, dtype=np.int32), mask=r.random(n) < 0.2)},  # row ids
}


def check(key, beside, asc, first):
    cols = {**beside, "k": key} if first else {"k": key, **beside}
    t = pa.table(cols)
    exp = stable_order([(key, none(len(key)))], [asc])
    assert_tables_equal(run_sort(t, ["k"], [asc]), t.take(pa.array(exp)), sort_by=None)


@pytest.mark.parametrize("beside", list(BESIDE))
@pytest.mark.parametrize("kind", ["random", "few", "u64", "i32", "u8", "one"])
def test_rows_beside_a_key(kind, beside):
    rng = np.random.default_rng(len(beside))
    n = N if kind != "u64" else 1 << 21
    key = {
        "random": lambda: rng.integers(-2**63, 2**63 - 1, n),
        "few": lambda: rng.integers(0, 1000, n) * 2**40 - 2**45,
        "u64": lambda: rng.integers(0, 2**64 - 1, n, dtype=np.uint64),
        "i32": lambda: rng.integers(-2**31, 2**31, n).astype(np.int32),
        "u8": lambda: rng.integers(0, 256, n).astype(np.uint8),
        "one": lambda: np.full(n, -7),
    }[kind]()
    for asc in (True, False):
        check(key, BESIDE[beside](rng, n), asc, first=asc)


@pytest.mark.parametrize("beside", ["i64", "wide"])
@pytest.mark.parametrize("cluster", [2, 12, 13, 257, 4096, 4097])
def test_clusters_of_leading_bits(cluster, beside):
    """Rows that agree in their leading 48 bits, half of them fully equal."""
    rng = np.random.default_rng(cluster)
    v = rng.integers(-2**62, 2**62, N)
    at = np.flatnonzero(np.arange(N) % STRIDE)[:: max(1, N // 20_000)][:cluster]
    v[at] = (v[5] & ~np.int64(0xFFFF)) | rng.integers(0, 1 << 16, cluster)
    v[at[::2]] = v[5]
    check(v, BESIDE[beside](rng, N), cluster % 2 == 0, first=False)
