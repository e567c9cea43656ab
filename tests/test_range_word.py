"""Where a row's 16-byte string range starts in its column: the helper
`range_word` of legate-dataframe_b200/csrc/radix.cu, which move_ranges indexes
with, compiled as host C++ and checked around the rows from which twice the row
number passes 32 bits."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
RADIX = ROOT / "legate-dataframe_b200" / "csrc" / "radix.cu"

DRIVER = r"""
#include <cstdint>
#include <cstdio>
#define __host__
#define __device__
#define __forceinline__ inline
#include "range_word.inc"
int main()
{
  const int32_t rows[] = {0, 1, 1000, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, 2147483646};
  for (int32_t r : rows)
    if (range_word(r) != static_cast<int64_t>(r) + r) return 1;
  std::puts("ok");
  return 0;
}
"""


def test_range_word_of_high_rows(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = RADIX.read_text()
    a = src.index("__host__ __device__ __forceinline__ int64_t range_word")
    (tmp_path / "range_word.inc").write_text(src[a:src.index("}\n", a) + 2])
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-fsanitize=undefined", "-fno-sanitize-recover", "-o", tmp_path / "t",
                    tmp_path / "t.cpp"], check=True)
    assert subprocess.run([tmp_path / "t"], capture_output=True, text=True).stdout == "ok\n"
    move = src[src.index("void move_ranges("):]
    assert "sp + range_word(row[k])" in move[:move.index("\n}\n")]
