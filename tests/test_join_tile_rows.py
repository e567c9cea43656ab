"""Output rows of one probe tile of a join with repeated build keys, checked on
the CPU: the helpers `wide_tile_rows` and `tile_row` of
legate-dataframe_b200/csrc/join.cu are compiled as host C++ and run on match
counts whose sums reach and pass 2^32, and every kernel member that holds such
a sum is 64 bits wide."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
JOIN = ROOT / "legate-dataframe_b200" / "csrc" / "join.cu"

DRIVER = r"""
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>
#define __host__
#define __device__
#define __forceinline__ inline
constexpr int kProbeTile = 1024;
#include "tile_row.inc"

template <typename T>
bool check(const std::vector<uint64_t>& count, std::mt19937_64& rng)
{
  std::vector<T> excl(kProbeTile);
  uint64_t total = 0;
  for (int r = 0; r < kProbeTile; ++r) {
    excl[r] = static_cast<T>(total);
    total += count[r];
  }
  uint64_t before = 0;
  for (int r = 0; r < kProbeTile; before += count[r], ++r) {
    if (count[r] == 0) continue;
    const uint64_t at[3] = {before, before + rng() % count[r], before + count[r] - 1};
    for (uint64_t j : at)
      if (tile_row<T>(excl.data(), static_cast<T>(j)) != r) {
        std::printf("FAIL row %d of output %llu of %llu\n", r, (unsigned long long)j, (unsigned long long)total);
        return false;
      }
  }
  return true;
}

int main()
{
  if (wide_tile_rows(0) || wide_tile_rows(0xffffffffll) || !wide_tile_rows(0x100000000ll)) return 1;
  std::mt19937_64 rng(7);
  for (int it = 0; it < 300; ++it) {
    // per probe row: none, one, a few or up to 2^31 - 1 build rows
    std::vector<uint64_t> count(kProbeTile);
    uint64_t total = 0;
    for (auto& c : count) {
      const int kind = static_cast<int>(rng() % 4);
      c = kind == 0 ? 0 : kind == 1 ? 1 : kind == 2 ? rng() % 50 : it % 3 ? rng() % 4000 : rng() % 0x7fffffff;
      total += c;
    }
    if (it == 0) {  // exactly 2^32 rows: a 32-bit count of them is 0
      total = 0;
      for (auto& c : count) total += c = 1u << 22;
    }
    if (!check<uint64_t>(count, rng)) return 1;
    if (!wide_tile_rows(static_cast<int64_t>(total)) && !check<uint32_t>(count, rng)) return 1;
  }
  std::puts("ok");
  return 0;
}
"""


def test_tile_rows_beyond_32_bits(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = JOIN.read_text()
    a = src.index("inline bool wide_tile_rows")
    b = src.index("}\n", src.index("int tile_row(const T* excl, T j)")) + 2
    (tmp_path / "tile_row.inc").write_text(src[a:b])
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-fsanitize=address,undefined", "-fno-sanitize-recover", "-Wno-unknown-pragmas",
                    "-o", tmp_path / "t", tmp_path / "t.cpp"], check=True)
    assert subprocess.run([tmp_path / "t"], capture_output=True, text=True).stdout == "ok\n"
    matches = src[src.index("struct Matches {"):]
    assert re.search(r"int64_t\* tile_counts;", matches[:matches.index("};")])
    assert "m.tile_counts[tile] = total;" in src


@pytest.mark.gpu
def test_one_tile_of_more_than_2_32_output_rows():
    """1,024 probe rows (and one more in a second tile) on a key of 2^22 + 3
    build rows: each probe row's value comes out once per build row."""
    import pyarrow as pa
    import torch

    from legate_dataframe import LogicalColumn, LogicalTable
    from legate_dataframe.lib.join import JoinType, join

    n, m = 1025, (1 << 22) + 3
    one = torch.ones(n, dtype=torch.int8, device="cuda")
    v = (torch.arange(n, device="cuda") % 5).to(torch.int8)
    lhs = LogicalTable([LogicalColumn.from_torch(one, pa.int8()), LogicalColumn.from_torch(v, pa.int8())], ["k", "v"])
    rhs = LogicalTable([LogicalColumn.from_torch(one[:1].expand(m).contiguous(), pa.int8())], ["r"])
    res = join(lhs, rhs, lhs_keys=["k"], rhs_keys=["r"], join_type=JoinType.INNER, lhs_out_columns=["v"],
               rhs_out_columns=[])
    col = res.get_column("v")
    assert col.size == n * m
    got = col.data[: n * m].view(torch.int8)
    counts = [sum(int((part == x).sum()) for part in got.split(1 << 30)) for x in range(5)]
    assert counts == [int((v == x).sum()) * m for x in range(5)]
