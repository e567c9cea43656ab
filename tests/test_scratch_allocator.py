"""Scratch buffers carved from chunks of the caller's allocator (class Allocator
in legate-dataframe_b200/csrc/common.cuh and runtime.cu), compiled as host C++
over a counting allocator: what a loop's buffers take does not grow with its
iterations, live buffers never overlap whatever the order they are given back
in, a pool too small for a chunk still serves small buffers, and everything goes
back with the size that it was taken with."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "legate-dataframe_b200" / "csrc"

DRIVER = r"""
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <map>
#include <memory>
#include <random>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>
using cudaStream_t = void*;
enum { cudaSuccess = 0, LDF_ERR_OUT_OF_MEMORY = 3 };
struct ldf_allocator {
  void* ctx;
  void* (*allocate)(void*, size_t, void*);
  void (*deallocate)(void*, void*, size_t, void*);
};
inline int cudaMallocAsync(void**, size_t, cudaStream_t) { return 1; }
inline int cudaFreeAsync(void*, cudaStream_t) { return 1; }
inline int cudaGetLastError() { return 0; }
[[noreturn]] inline void fail(int, const std::string& m) { throw std::runtime_error(m); }
#include "allocator.inc"

struct Pool {
  size_t limit, now = 0, peak = 0;
  uintptr_t next = 4096;
  int wrong = 0;
  std::map<void*, size_t> live;
};
static void* take(void* ctx, size_t n, void*)
{
  Pool& p = *static_cast<Pool*>(ctx);
  if (p.now + n > p.limit) return nullptr;
  p.now += n;
  p.peak = std::max(p.peak, p.now);
  void* a = reinterpret_cast<void*>(p.next);
  p.next += n + 4096;
  p.live[a] = n;
  return a;
}
static void give(void* ctx, void* a, size_t n, void*)
{
  Pool& p = *static_cast<Pool*>(ctx);
  auto it = p.live.find(a);
  if (it == p.live.end() || it->second != n) ++p.wrong;
  if (it != p.live.end()) {
    p.now -= it->second;
    p.live.erase(it);
  }
}
#define CHECK(c) do { if (!(c)) { std::printf("FAIL %s, line %d\n", #c, __LINE__); std::exit(1); } } while (0)

static size_t loop_peak(int iterations)
{
  Pool pool{size_t(1) << 40};
  ldf_allocator a{&pool, take, give};
  {
    Allocator al(&a, nullptr);
    Buffer<int> kept(al, 100);
    Buffer<int> late;
    for (int i = 0; i < iterations; ++i) {
      Buffer<uint64_t> word(al, 900000), other(al, 800000);
      Buffer<uint32_t> perm(al, 1000000);
      if (i == 0) late = Buffer<int>(al, 1);  // made in the first round, kept to the end
      Buffer<uint8_t> big(al, 20000000);
      word = Buffer<uint64_t>(al, 500000);
    }
  }
  CHECK(pool.live.empty() && pool.wrong == 0);
  return pool.peak;
}

int main()
{
  const size_t few = loop_peak(2);
  CHECK(loop_peak(500) == few);

  for (int seed = 0; seed < 200; ++seed) {  // any order of taking and giving back
    std::mt19937_64 rng(seed);
    Pool pool{size_t(1) << 40};
    ldf_allocator a{&pool, take, give};
    {
      Allocator al(&a, nullptr);
      std::vector<std::unique_ptr<Buffer<char>>> b;
      std::map<char*, size_t> live;
      for (int i = 0; i < 400; ++i) {
        if (b.empty() || rng() % 5 < 3) {
          const size_t n = rng() % 4 == 0 ? rng() % (12u << 20) : rng() % 5000;
          b.push_back(std::make_unique<Buffer<char>>(al, n));
          char* p = b.back()->get();
          const size_t size = b.back()->bytes();
          auto up = live.lower_bound(p);
          CHECK(reinterpret_cast<uintptr_t>(p) % 256 == 0);
          CHECK(up == live.end() || p + size <= up->first);
          CHECK(up == live.begin() || std::prev(up)->first + std::prev(up)->second <= p);
          bool inside = false;
          for (auto& c : pool.live) {
            char* q = static_cast<char*>(c.first);
            inside = inside || (p >= q && p + size <= q + c.second);
          }
          CHECK(inside);
          live[p] = size;
        } else {
          const size_t k = rng() % 3 ? b.size() - 1 : rng() % b.size();
          live.erase(b[k]->get());
          b.erase(b.begin() + k);
        }
      }
    }
    CHECK(pool.live.empty() && pool.wrong == 0);
  }

  {  // no room for a chunk
    Pool pool{size_t(3) << 20};
    ldf_allocator a{&pool, take, give};
    {
      Allocator al(&a, nullptr);
      for (int i = 0; i < 10; ++i) {
        Buffer<char> x(al, 1000), y(al, 1 << 20), z(al, 500);
        CHECK(x.get() && y.get() && z.get());
      }
      bool threw = false;
      try {
        Buffer<char> w(al, 4 << 20);
      } catch (const std::runtime_error&) {
        threw = true;
      }
      CHECK(threw);
    }
    CHECK(pool.live.empty() && pool.wrong == 0);
  }
  std::puts("ok");
  return 0;
}
"""


def test_scratch_allocator(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    head, body = (CSRC / "common.cuh").read_text(), (CSRC / "runtime.cu").read_text()
    cls = head[head.index("class Allocator {"):]
    cls = cls[:cls.index("\n// ----", cls.index("class Buffer"))]
    end = body.index("\n}\n", body.index("Allocator::~Allocator()")) + 3
    start = min(body.index(f"void* Allocator::{f}(") for f in ("allocate", "try_allocate") if f"void* Allocator::{f}(" in body)
    (tmp_path / "allocator.inc").write_text(cls + body[start:end])
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=address,undefined", "-fno-sanitize-recover", "-o",
                    tmp_path / "t", tmp_path / "t.cpp"], check=True)
    res = subprocess.run([tmp_path / "t"], capture_output=True, text=True)
    assert res.stdout == "ok\n", res.stdout + res.stderr
