"""Snappy pages of several 64 KB fragments (decoded a warp per fragment)
through the C ABI: streams of Arrow's compressor at the edges of fragments and
stream segments, hand-made streams whose elements cross the fragments (decoded
again by the per-page kernels), and malformed ones."""

import ctypes

import numpy as np
import pyarrow as pa
import pytest
import torch

pytestmark = pytest.mark.gpu


def decode(streams, values_per_page, physical, ldf_type, sizes):
    """The column held by one PLAIN data page per stream."""
    from legate_dataframe import _native as N

    pages = (N.ldf_parquet_page * len(streams))()
    blob, row = b"", 0
    for p, (st, nv, u) in enumerate(zip(streams, values_per_page, sizes)):
        q = pages[p]
        q.offset, q.compressed, q.uncompressed, q.row0, q.num_values = len(blob), len(st), u, row, nv
        q.kind, q.encoding, q.codec, q.dict = N.LDF_PQ_DATA_V1, 0, N.LDF_PQ_SNAPPY, -1
        blob += st
        row += nv
    file = torch.from_numpy(np.frombuffer(blob, np.uint8).copy()).cuda()
    alloc, out = N.TorchAllocator(torch.device("cuda", 0)), (N.ldf_column * 1)()
    N.check(N.lib().ldf_b200_parquet_decode(file.data_ptr(), len(blob), pages, len(streams), N.int32_array([physical]),
                                            N.int32_array([ldf_type]), N.int32_array([0]), 1, row, out,
                                            ctypes.byref(alloc.struct), ctypes.c_void_p(N.current_stream_handle())))
    from legate_dataframe import LogicalColumn

    t = {N.LDF_INT64: pa.int64(), N.LDF_STRING: pa.string()}[ldf_type]
    return LogicalColumn.from_c(out[0], t, alloc).to_arrow()


def varint(n):
    b = bytearray()
    while n > 127:
        b.append(n & 127 | 128)
        n >>= 7
    return bytes(b + bytes([n]))


def literal(data):
    n = len(data) - 1
    return (bytes([n << 2]) if n < 60 else bytes([62 << 2]) + n.to_bytes(3, "little")) + data


def copy(offset, n):
    assert 1 <= n <= 64
    return bytes([(n - 1) << 2 | 3]) + offset.to_bytes(4, "little")


def int64_pages(rng, sizes):
    kinds = [lambda n: rng.integers(-2**40, 2**40, n), lambda n: rng.integers(0, 50, n),
             lambda n: np.arange(n) // 7, lambda n: np.zeros(n, np.int64),
             lambda n: rng.integers(-2**63, 2**63 - 1, n)]
    return [kinds[i % len(kinds)](n // 8).astype(np.int64) for i, n in enumerate(sizes)]


def test_int64_pages_at_fragment_edges():
    from legate_dataframe import _native as N

    rng = np.random.default_rng(3)
    sizes = [s for s in (65536, 65544, 131072, 131080, 196608, 1 << 20, (1 << 20) + 8, 3_000_000) for _ in range(5)]
    vals = int64_pages(rng, sizes)
    streams = [pa.compress(v.tobytes(), codec="snappy", asbytes=True) for v in vals]
    got = decode(streams, [len(v) for v in vals], N.LDF_PQ_INT64, N.LDF_INT64, sizes)
    assert np.array_equal(got.to_numpy(), np.concatenate(vals))


def crossing_stream(rng, n):
    """Elements and copies that pay no heed to the fragments, and the bytes."""
    data, st = bytearray(rng.integers(0, 256, 70_001, dtype=np.uint8).tobytes()), bytearray(varint(n))
    st += literal(bytes(data))
    while len(data) < n:
        m = int(min(n - len(data), rng.integers(1, 65)))
        if rng.random() < 0.5:
            off = int(rng.integers(1, len(data) + 1))
            st += copy(off, m)
            for _ in range(m):
                data.append(data[-off])
        else:
            piece = rng.integers(0, 256, m, dtype=np.uint8).tobytes()
            st += literal(piece)
            data += piece
    return bytes(st), bytes(data)


def test_streams_that_cross_fragments():
    from legate_dataframe import _native as N

    rng = np.random.default_rng(4)
    n = 200_000
    crossing, plain = crossing_stream(rng, n)
    one = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
    good = np.arange(n // 8)
    fine = pa.compress(good.tobytes(), codec="snappy", asbytes=True)
    # bytes behind the last element are left alone
    streams = [crossing, varint(n) + literal(one), fine, fine + literal(b"more")]
    got = decode(streams, [n // 8] * 4, N.LDF_PQ_INT64, N.LDF_INT64, [n] * 4)
    exp = np.concatenate([np.frombuffer(plain, np.int64), np.frombuffer(one, np.int64), good, good])
    assert np.array_equal(got.to_numpy(), exp)


def test_byte_array_stream_that_crosses_fragments():
    from legate_dataframe import _native as N

    words = [f"value {i * 7919 % 10007:05d}{'x' * (i % 23)}" for i in range(12_000)]
    data = b"".join(len(w).to_bytes(4, "little") + w.encode() for w in words)
    crossing = varint(len(data)) + literal(data)
    fine = pa.compress(data, codec="snappy", asbytes=True)
    got = decode([crossing, fine, crossing], [len(words)] * 3, N.LDF_PQ_BYTE_ARRAY, N.LDF_STRING, [len(data)] * 3)
    assert got.to_pylist() == words * 3


@pytest.mark.parametrize("how", ["offset", "zero_offset", "short", "length"])
def test_malformed_stream_of_several_fragments(how):
    from legate_dataframe import _native as N

    n = 160_000
    base = np.arange(n // 8).tobytes()
    fine = pa.compress(base, codec="snappy", asbytes=True)
    if how == "offset":
        bad = varint(n) + literal(base[:100]) + copy(101, 64) + literal(base[164:])
    elif how == "zero_offset":
        bad = varint(n) + literal(base[:100]) + copy(0, 64) + literal(base[164:])
    elif how == "short":
        bad = fine[:-5]
    else:
        bad = varint(n + 8) + fine[len(varint(n)):]
    with pytest.raises(ValueError, match="Parquet page 1: a Snappy stream is malformed"):
        decode([fine, bad], [n // 8] * 2, N.LDF_PQ_INT64, N.LDF_INT64, [n] * 2)


@pytest.mark.parametrize("version", ["1.0", "2.0"])
@pytest.mark.parametrize("compression", ["snappy", "none"])
@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("n", [255, 256, 20_000, 100_003])
def test_plain_strings(tmp_path, n, nulls, compression, version):
    """PLAIN byte-array pages (length prefixes ranked per 4 KB segment): empty
    strings, strings of several segments, strings that end at a segment."""
    import pyarrow.parquet as pq

    from legate_dataframe.lib.parquet import parquet_read

    rng = np.random.default_rng(n)
    words = ["", "a", "xyz" * 7, "s" * 4088, "q" * 4092, "long " * 2500] + [f"w{i}" * (i % 9) for i in range(500)]
    w = rng.integers(0, len(words), n)
    w[rng.random(n) < 0.995] %= 3
    t = pa.table({"s": pa.array([words[i] for i in w], mask=rng.random(n) < 0.3 if nulls else None), "i": np.arange(n)})
    path = tmp_path / "t.parquet"
    pq.write_table(t, path, use_dictionary=False, compression=compression, data_page_version=version,
                   data_page_size=200_000)
    assert parquet_read(str(path)).to_arrow().equals(t)


def test_truncated_plain_strings():
    from legate_dataframe import _native as N

    data = b"".join(len(w).to_bytes(4, "little") + w for w in [b"value"] * 20_000)
    for cut in (1, 5, 9_000):
        st = pa.compress(data[:-cut], codec="snappy", asbytes=True)
        with pytest.raises(ValueError, match="Parquet page 0: the page's values are truncated"):
            decode([st], [20_000], N.LDF_PQ_BYTE_ARRAY, N.LDF_STRING, [len(data) - cut])
