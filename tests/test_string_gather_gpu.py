"""String columns through a gather (a sort's order) at the edges of its tiles,
and from a column whose characters lie beyond 2^32."""

import numpy as np
import pyarrow as pa
import pytest

from ldf_testing import assert_tables_equal
from test_sort_gpu import run_sort

pytestmark = pytest.mark.gpu


def strings(rng, n, longest):
    return pa.array([None if rng.random() < 0.1 else "x" * int(rng.integers(0, longest)) + str(i) for i in range(n)])


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 1024, 20_001])
@pytest.mark.parametrize("longest", [1, 9, 300])
def test_tile_edges(n, longest):
    rng = np.random.default_rng(n + longest)
    key = rng.permutation(n)
    t = pa.table({"k": key, "s": strings(rng, n, longest), "f": rng.normal(size=n)})
    assert_tables_equal(run_sort(t, ["k"], [True]), t.take(pa.array(np.argsort(key))), sort_by=None)


def test_characters_beyond_32_bits():
    """2^32 + 1 KB characters, of which the rows name a few at either end."""
    import torch

    from legate_dataframe import _native as N
    from legate_dataframe import LogicalTable
    from legate_dataframe.lib.core.column import LogicalColumn
    from legate_dataframe.lib.sort import sort

    total = (1 << 32) + 1024
    n = 700
    rng = np.random.default_rng(3)
    chars = torch.zeros(total, dtype=torch.uint8, device="cuda")
    ends = torch.from_numpy(rng.integers(97, 123, 2048).astype(np.uint8)).cuda()
    chars[:1024], chars[-1024:] = ends[:1024], ends[1024:]
    text = ends.cpu().numpy().tobytes().decode()
    lo = rng.integers(0, 1000, n)
    ln = rng.integers(0, 24, n)
    far = rng.random(n) < 0.5
    start = lo + np.where(far, total - 1024, 0)
    ranges = torch.from_numpy(np.stack([start, start + ln - 1], 1).astype(np.int64)).cuda().view(torch.uint8).reshape(-1)
    s = LogicalColumn(pa.string(), N.LDF_STRING, n, ranges, None, chars, 0, total)
    key = rng.permutation(n)
    exp = [text[a + 1024 * b : a + 1024 * b + c] for a, b, c in zip(lo, far, ln)]
    k = LogicalColumn.from_arrow(pa.array(key))
    out = sort(LogicalTable([k, s], ["k", "s"]), ["k"])
    assert out["s"].to_arrow().to_pylist() == [exp[i] for i in np.argsort(key)]
