"""Which passes of the radix sort prefetch the rows' values into L2: the first
pass of a sort whose rows travel whole reads the caller's own column, which is
prefetched only when it is device memory.  The rule (`prefetch_values` in
legate-dataframe_b200/csrc/radix.cu) is compiled as host C++; on the GPU such
a sort of columns in pinned host memory matches numpy."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
RADIX = ROOT / "legate-dataframe_b200" / "csrc" / "radix.cu"

DRIVER = r"""
#include <cstddef>
#include <cstdio>
int g_first = 1;
int prefetch_first_pass() { return g_first; }
#include "rule.inc"
int main()
{
  int device = 0, host = 0, asked = 0;
  auto on_device = [&](const void* p) { ++asked; return p == &device; };
  if (prefetch_values(0, &host, on_device) != 0 || prefetch_values(0, &device, on_device) != 1 || asked != 2) return 1;
  if (prefetch_values(0, nullptr, on_device) != 0 || asked != 2) return 2;
  if (prefetch_values(1, &host, on_device) != 1 || prefetch_values(3, nullptr, on_device) != 1 || asked != 2) return 3;
  g_first = 0;  // LDF_B200_L2_PREFETCH_FIRST=0
  if (prefetch_values(0, &device, on_device) != 0 || prefetch_values(1, &device, on_device) != 1) return 4;
  std::puts("ok");
  return 0;
}
"""


def test_first_pass_asks_where_the_values_are(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = RADIX.read_text()
    a = src.index("template <typename F>\nint prefetch_values(")
    (tmp_path / "rule.inc").write_text(src[a:src.index("\n}\n", a) + 3])
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-o", tmp_path / "t", tmp_path / "t.cpp"], check=True)
    assert subprocess.run([tmp_path / "t"], capture_output=True, text=True).stdout == "ok\n"
    assert "if (a.pf_vals && a.vals_in) l2_prefetch_bulk(a.vals_in," in src
    assert "a.pf_vals    = prefetch_values(k, first_vals, on_device);" in src


@pytest.mark.gpu
@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("pinned", ["key", "value", "both"])
def test_whole_row_sort_of_pinned_columns(width, pinned):
    import ctypes

    import torch

    from legate_dataframe import _native as N

    n = (1 << 21) + 77
    rng = np.random.default_rng(width)
    key = rng.integers(-2**62, 2**62, n)
    key[::5] = key[0]
    val = rng.integers(-2**31, 2**31, n).astype(np.int32 if width == 4 else np.int64)

    def place(x, host):
        t = torch.from_numpy(x)
        return t.pin_memory() if host else t.cuda()

    k, v = place(key, pinned != "value"), place(val, pinned != "key")
    table = (N.ldf_column * 2)()
    for col, t, ty in ((table[0], k, N.LDF_INT64), (table[1], v, N.LDF_INT32 if width == 4 else N.LDF_INT64)):
        col.type, col.nullable, col.size, col.data = ty, 0, n, t.data_ptr()
    alloc = N.TorchAllocator(N.require_cuda())
    out = (N.ldf_column * 2)()
    torch.cuda.synchronize()
    N.check(N.lib().ldf_b200_sort(table, 2, N.int32_array([0]), (ctypes.c_uint8 * 1)(1), 1, 1, 1, -(2**63), out,
                                  ctypes.byref(alloc.struct), ctypes.c_void_p(N.current_stream_handle())))
    order = np.argsort(key, kind="stable")
    got = [alloc.adopt(out[j].data).cpu().numpy()[: n * w].view(t) for j, w, t in ((0, 8, np.int64), (1, width, val.dtype))]
    assert np.array_equal(got[0], key[order])
    assert np.array_equal(got[1], val[order])
