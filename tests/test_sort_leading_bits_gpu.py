"""Sorts on the leading bits of the fused key word (2^21 rows and more), with
the ties among them ordered afterwards, and fused words of nullable and float
keys, against numpy's stable sort of the same order."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from test_sort_gpu import run_sort

pytestmark = pytest.mark.gpu

N = (1 << 21) + 5
STRIDE = -(-N // (1 << 17))  # every STRIDE-th row is sampled


def stable_order(columns, asc, nulls_at_end=True):
    """Row order by (values, mask) columns, most significant first."""
    perm = np.arange(len(columns[0][0]))
    for (v, null), a in reversed(list(zip(columns, asc))):
        x = np.where(null | (v != v), 0, v).astype(v.dtype)[perm]  # nulls and NaNs: placed by class below
        if not a:  # descending, ties in order: sort the reversed rows and reverse
            o = (len(x) - 1 - np.argsort(x[::-1], kind="stable"))[::-1]
        else:
            o = np.argsort(x, kind="stable")
        perm = perm[o]
        x = v[perm]
        cls = null[perm] * 2
        if x.dtype.kind == "f":
            cls = np.where(null[perm], 2, np.isnan(x) * 1)
        perm = perm[np.argsort(cls if nulls_at_end else 2 - cls, kind="stable")]
    return perm


def check(columns, asc, nulls_at_end=True, limit=None):
    names = [f"k{i}" for i in range(len(columns))]
    t = pa.table({n: pa.array(v, mask=m if m.any() else None) for n, (v, m) in zip(names, columns)}
                 | {"row": np.arange(len(columns[0][0]), dtype=np.int32)})
    res = run_sort(t, names, asc, nulls_at_end, limit=limit)
    exp = stable_order(columns, asc, nulls_at_end)
    exp = exp if limit is None else exp[:limit]
    assert np.array_equal(res.column("row").to_numpy(), exp)
    assert_tables_equal(res, t.take(pa.array(exp)), sort_by=None)


def none(n=N):
    return np.zeros(n, bool)


@pytest.mark.parametrize("asc", [True, False])
@pytest.mark.parametrize("cluster", [0, 2, 12, 13, 60, 3000, 4096, 4097, 9000])
def test_clusters_of_leading_bits(cluster, asc):
    """Random keys and a group of rows that agree in their leading 48 bits, at
    rows that the sample does not see: ordered by a thread, by a block, or, over
    4,096 rows, by sorting the whole word.  Half of them are fully equal."""
    rng = np.random.default_rng(cluster)
    v = rng.integers(-2**62, 2**62, N)
    at = np.flatnonzero(np.arange(N) % STRIDE)[:: max(1, N // 20_000)][:cluster]
    assert len(at) == cluster
    v[at] = (v[5] & ~np.int64(0xFFFF)) | rng.integers(0, 1 << 16, cluster)
    v[at[::2]] = v[5]
    check([(v, none())], [asc])


@pytest.mark.parametrize("kind", ["duplicates", "narrow", "skewed", "limit"])
def test_other_distributions(kind):
    rng = np.random.default_rng(7)
    if kind == "duplicates":  # every key many times: no bits to drop
        v = rng.integers(0, 1000, N) * 2**40
    elif kind == "narrow":  # 45 bits of range
        v = 1_600_000_000_000_000 + rng.integers(0, 2**45, N)
    elif kind == "skewed":  # most rows in one 16-bit corner
        v = np.where(rng.random(N) < 0.7, rng.integers(0, 2**16, N), rng.integers(-2**60, 2**60, N))
    else:
        v = rng.integers(-2**63, 2**63 - 1, N)
    check([(v, none())], [True], limit=1000 if kind == "limit" else None)


@pytest.mark.parametrize("n", [20_000, N])
@pytest.mark.parametrize("nulls_at_end", [True, False])
@pytest.mark.parametrize("asc", [[True, False], [False, True]])
def test_nullable_and_float_keys(n, nulls_at_end, asc):
    rng = np.random.default_rng(n)
    f = rng.normal(size=n) * 10.0 ** rng.integers(-5, 5, n)
    f[::97], f[1::97], f[2::97], f[3::97] = np.nan, np.inf, -np.inf, -0.0
    i = rng.integers(-2**20, 2**20, n)
    g = (rng.integers(-4, 4, n) / 2).astype(np.float32)
    g[::11] = np.nan
    check([(f, rng.random(n) < 0.1)], asc[:1], nulls_at_end)
    check([(i, rng.random(n) < 0.3), (g, rng.random(n) < 0.3)], asc, nulls_at_end)
    check([(g, none(n)), (f, rng.random(n) < 0.1)], asc, nulls_at_end)  # over 72 bits: pass by pass
    check([(np.zeros(n, np.int64), np.ones(n, bool)), (i, none(n))], asc, nulls_at_end)
