"""PLAIN string pages of several hundred MB: their length prefixes are ranked a
round of 128 MB at a time, so that the scratch does not grow with the file."""

import numpy as np
import pyarrow as pa
import pyarrow.parquet as pq
import pytest

pytestmark = pytest.mark.gpu


def strings(n, length, nulls):
    chars = np.random.default_rng(n).integers(97, 123, n * length, dtype=np.uint8)
    lens = np.full(n, length, np.int32)
    lens[::7] = 0
    off = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=off[1:])
    a = pa.Array.from_buffers(pa.string(), n, [None, pa.py_buffer(off), pa.py_buffer(chars)])
    return pa.array(a.to_pylist(), mask=np.arange(n) % 5 == 0) if nulls else a


@pytest.mark.parametrize("compression", ["none", "snappy"])
def test_scratch_of_plain_strings_is_bounded(tmp_path, compression):
    import torch

    from legate_dataframe.lib.parquet import parquet_read

    t = pa.table({"s": strings(4_000_000, 100, False)})
    pq.write_table(t, tmp_path / "f", use_dictionary=False, compression=compression)
    parquet_read(tmp_path / "f")  # warm: the allocator and the kernels
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    res = parquet_read(tmp_path / "f")
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - before
    assert res.to_arrow().column("s").combine_chunks().cast(pa.string()).equals(t.column("s").combine_chunks())
    # the file, the decompressed pages, the characters (360 MB each) and 72 bytes a row, besides 8 bytes for
    # each of a round's
    assert peak < 3 * (360 << 20) + 72 * 4_000_000 + 8 * (128 << 20) + (64 << 20), peak


@pytest.mark.parametrize("rows_per_page, rounds", [(2000, "many pages"), (1 << 20, "few pages")])
def test_rounds_match_pyarrow(tmp_path, rows_per_page, rounds):
    from legate_dataframe.lib.parquet import parquet_read

    t = pa.table({"a": strings(600_000, 300, True), "b": strings(600_000, 40, False), "i": np.arange(600_000)})
    pq.write_table(t, tmp_path / "f", use_dictionary=False, compression="none", row_group_size=200_000,
                   data_page_size=rows_per_page * 300)
    res = parquet_read(tmp_path / "f").to_arrow()
    for name in t.column_names:
        got = res.column(name).combine_chunks()
        assert (got.cast(pa.string()) if name != "i" else got).equals(t.column(name).combine_chunks())
