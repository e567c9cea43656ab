"""Buffers that a groupby takes from and returns to the caller's allocator: the
outputs of a small input are as large as its groups need, and every buffer goes
back with the size that it was taken with."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ledger_allocator(N, torch):
    live, wrong = {}, []

    def alloc(ctx, nbytes, stream):
        t = torch.empty(int(nbytes), dtype=torch.uint8, device="cuda")
        live[t.data_ptr()] = (int(nbytes), t)
        return t.data_ptr()

    def free(ctx, ptr, nbytes, stream):
        size, _ = live.pop(ptr)
        if size != int(nbytes):
            wrong.append((size, int(nbytes)))

    cbs = N.ALLOC_FN(alloc), N.DEALLOC_FN(free)
    return N.ldf_allocator(None, *cbs), cbs, live, wrong


@pytest.mark.parametrize("n, groups", [(1000, 7), (131072, 1), (131072, 131072), (131073, 10)])
@pytest.mark.parametrize("string", [False, True])
def test_groupby_outputs_are_sized_to_the_groups(n, groups, string):
    import pyarrow as pa
    import torch

    from legate_dataframe import LogicalTable
    from legate_dataframe import _native as N

    key = np.arange(n) % groups
    t = LogicalTable.from_arrow(pa.table({"k": [f"key{x}" for x in key.tolist()] if string else key, "v": np.ones(n)}))
    k, v = t.get_column("k"), t.get_column("v")
    cols = (N.ldf_column * 2)()
    for c, col in zip(cols, (k, v)):
        c.type, c.nullable, c.size, c.data = col.ldf_type, 0, n, col.data.data_ptr()
        if col.ldf_type == N.LDF_STRING:
            c.chars, c.chars_base, c.num_chars = col.chars.data_ptr(), col.chars_base, col.num_chars
    agg = (N.ldf_aggregation * 1)()
    agg[0].in_col, agg[0].kind, agg[0].out_type = 1, N.LDF_AGG["sum"], N.LDF_FLOAT64
    struct, cbs, live, wrong = ledger_allocator(N, torch)
    out = (N.ldf_column * 2)()
    L, stream = N.lib(), ctypes.c_void_p(N.current_stream_handle())
    N.check(L.ldf_b200_groupby_aggregation(cols, 2, N.int32_array([0]), 1, agg, 1, out, ctypes.byref(struct), stream))
    assert [c.size for c in out] == [groups, groups]
    assert live[out[1].data][0] == (8 * groups + 255) // 256 * 256
    for c in out:
        N.check(L.ldf_b200_free_column(ctypes.byref(c), ctypes.byref(struct), stream))
    torch.cuda.synchronize()
    assert wrong == [] and live == {}


def test_sort_scratch_does_not_grow_with_string_length():
    """20,000 distinct strings that differ behind one of two prefixes: the scratch
    of the chunk after chunk ranking at 1,600 bytes is that at 64."""
    import pyarrow as pa
    import torch

    from legate_dataframe import LogicalTable
    from legate_dataframe import _native as N

    def scratch_peak(prefix):
        n = 20_000
        order = np.random.default_rng(prefix).permutation(n)
        col = LogicalTable.from_arrow(pa.table({"k": ["pq"[x % 2] * prefix + f"{x:06d}" for x in order.tolist()]})).get_column("k")
        c = (N.ldf_column * 1)()
        c[0].type, c[0].nullable, c[0].size, c[0].data = N.LDF_STRING, 0, n, col.data.data_ptr()
        c[0].chars, c[0].chars_base, c[0].num_chars = col.chars.data_ptr(), col.chars_base, col.num_chars
        struct, (take, give), live, wrong = ledger_allocator(N, torch)
        peak = 0

        def counted(ctx, nbytes, stream):
            nonlocal peak
            p = take(ctx, nbytes, stream)
            peak = max(peak, sum(size for size, _ in live.values()))
            return p

        counted_cb = N.ALLOC_FN(counted)
        struct = N.ldf_allocator(None, counted_cb, give)
        out = (N.ldf_column * 1)()
        stream = ctypes.c_void_p(N.current_stream_handle())
        N.check(N.lib().ldf_b200_sort(c, 1, N.int32_array([0]), (ctypes.c_uint8 * 1)(1), 1, 1, 1, -(2**63), out,
                                      ctypes.byref(struct), stream))
        got = np.frombuffer(live[out[0].chars][1].cpu().numpy().tobytes()[: out[0].num_chars], "S%d" % (prefix + 6))
        assert np.array_equal(got, np.sort(got)) and len(np.unique(got)) == n
        held = sum(live[p][0] for p in (out[0].data, out[0].chars))
        N.check(N.lib().ldf_b200_free_column(ctypes.byref(out[0]), ctypes.byref(struct), stream))
        assert live == {} and wrong == []
        return peak - held

    assert scratch_peak(1600) <= scratch_peak(64) + (1 << 20)
