"""The thread-block cluster of a small groupby is no larger than the device can
hold: the rule (`fit_cluster` in legate-dataframe_b200/csrc/groupby.cu) compiled
as host C++, with devices that hold 16, 8, one or no CTA of a cluster."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
GROUPBY = ROOT / "legate-dataframe_b200" / "csrc" / "groupby.cu"

DRIVER = r"""
#include <cstdio>
#include "rule.inc"
int main()
{
  const unsigned holds[] = {16, 8, 1, 0}, asked[] = {1, 2, 5, 5};
  for (int q = 0; q < 4; ++q) {
    unsigned calls = 0;
    const unsigned got = fit_cluster(16, [&](unsigned c) { ++calls; return c <= holds[q] ? 1 : 0; });
    if (got != holds[q] || calls != asked[q]) return 1 + q;
  }
  if (fit_cluster(16, [](unsigned c) { return c <= 4 ? 3 : -1; }) != 4) return 5;
  std::puts("ok");
  return 0;
}
"""


def test_cluster_fits_the_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    src = GROUPBY.read_text()
    a = src.index("template <typename F>\nunsigned fit_cluster(")
    (tmp_path / "rule.inc").write_text(src[a:src.index("\n}\n", a) + 3])
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-o", tmp_path / "t", tmp_path / "t.cpp"], check=True)
    assert subprocess.run([tmp_path / "t"], capture_output=True, text=True).stdout == "ok\n"
    body = src[src.index("bool small_groupby("):]
    # nothing is allocated before a call without a cluster goes to the general plan
    assert body.index("if (most == 0) return false;") < body.index("Buffer<")
