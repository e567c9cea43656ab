"""Reading a file into pinned host memory and on to the device
(legate-dataframe_b200/csrc/file_read.cu), on the CPU: the source is compiled as
host C++ against a stand-in for the CUDA calls, called with the per-thread
stream's handle, which is another stream in every thread.  Every byte must have
been copied when the call returns, behind the caller's earlier work; failed
reads give their errno."""

import errno
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "legate-dataframe_b200" / "csrc" / "file_read.cu"
PIECE = 2 << 20

FAKE = r"""
#pragma once
#include <cstdint>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <thread>
#include <tuple>
#include <utility>
#include <vector>
using cudaStream_t = void*;
enum cudaError_t { cudaSuccess = 0, cudaErrorUnknown = 1 };
enum { cudaMemcpyHostToDevice = 1, LDF_ERR_CUDA = 2 };
using Stream = std::pair<cudaStream_t, std::thread::id>;  // the handle 2 is one stream per thread
struct Copy {
  Stream on;
  void* dst;
  const void* src;
  size_t n;
};
struct Event {
  Stream on;
};
using cudaEvent_t = Event*;
enum { cudaEventDisableTiming = 2 };
inline std::mutex g_mu;
inline std::vector<Copy> g_queued;  // copies not yet done
inline std::vector<Stream> g_behind;  // streams that wait for the caller's earlier work
inline Stream g_caller;
inline int g_early = 0, g_events = 0;
inline Stream stream_of(cudaStream_t s)
{
  return {s, s == reinterpret_cast<cudaStream_t>(2) ? std::this_thread::get_id() : std::thread::id{}};
}
inline void run(const Stream& on)
{
  std::lock_guard<std::mutex> lock(g_mu);
  for (const Copy& c : g_queued)
    if (c.on == on) std::memcpy(c.dst, c.src, c.n);
}
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = new Event; ++g_events; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; --g_events; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->on = stream_of(s); return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int)
{
  if (e->on == g_caller) g_behind.push_back(stream_of(s));
  return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, int, cudaStream_t s)
{
  std::lock_guard<std::mutex> lock(g_mu);
  const Stream on = stream_of(s);
  g_queued.push_back(Copy{on, dst, src, n});
  bool behind = on == g_caller;
  for (const Stream& b : g_behind) behind = behind || b == on;
  if (!behind) ++g_early;
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(stream_of(s)); return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) { run(e->on); return cudaSuccess; }
#define LDF_REQUIRE(c, m) do { if (!(c)) throw std::runtime_error(m); } while (0)
#define LDF_CUDA(e) do { if ((e) != cudaSuccess) throw std::runtime_error("cuda"); } while (0)
namespace ldf {
inline cudaStream_t staging_stream() { return reinterpret_cast<cudaStream_t>(16); }
[[noreturn]] inline void fail(int, const char* m) { throw std::runtime_error(m); }
inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
}
"""

DRIVER = r"""
#include "file_read.cu"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv)
{
  const int64_t n = std::atoll(argv[2]);
  const cudaStream_t per_thread = reinterpret_cast<cudaStream_t>(2);
  g_caller = stream_of(per_thread);
  std::vector<uint8_t> host(n + 1, 1), dev(n + 1, 2);
  const int e = ldf::read_file(argv[1], n, host.data(), dev.data(), per_thread);
  std::fprintf(stderr, "%d %d\n", e, g_early + g_events);
  if (e == 0) std::fwrite(dev.data(), 1, n, stdout);
  return dev[n] == 2 && host[n] == 1 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def reader(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("file_read")
    (d / "scan.cuh").write_text(FAKE)
    (d / "file_read.cu").write_text(SRC.read_text())
    (d / "t.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=address,undefined", "-pthread", "-o", d / "t", d / "t.cpp"],
                   check=True)

    def read(path, n):
        res = subprocess.run([d / "t", os.fspath(path), str(n)], capture_output=True, timeout=120)
        assert res.returncode == 0, res.stderr.decode()
        err, early = map(int, res.stderr.split())
        return err, early, res.stdout

    return read


@pytest.mark.parametrize("n", [0, 1, PIECE - 1, PIECE, PIECE + 1, 9 * PIECE + 12345, 40 * PIECE])
def test_copies_are_complete(reader, tmp_path, n):
    data = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8).tobytes()
    (tmp_path / "f").write_bytes(data)
    err, early, got = reader(tmp_path / "f", n)
    assert (err, early) == (0, 0)
    assert got == data


def test_failed_reads(reader, tmp_path):
    assert reader(tmp_path / "missing", 10)[0] == errno.ENOENT
    assert reader(tmp_path, 10)[0] == errno.EISDIR
    (tmp_path / "short").write_bytes(b"x" * (3 * PIECE + 5))
    assert reader(tmp_path / "short", 3 * PIECE + 6)[0] == errno.EIO
    assert reader(tmp_path / "short", 30 * PIECE)[0] == errno.EIO


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, PIECE, 20 * PIECE + 7])
@pytest.mark.parametrize("per_thread", [False, True])
def test_read_file_on_the_gpu(tmp_path, n, per_thread):
    import ctypes

    import torch

    from legate_dataframe import _native as N

    data = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    (tmp_path / "f").write_bytes(data.tobytes())
    host = torch.empty(n, dtype=torch.uint8, pin_memory=True)
    dev = torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    err = ctypes.c_int32(-1)
    stream = 2 if per_thread else N.current_stream_handle()  # 2: cudaStreamPerThread
    N.check(N.lib().ldf_b200_read_file(os.fsencode(tmp_path / "f"), n, host.data_ptr(), dev.data_ptr(),
                                       ctypes.byref(err), ctypes.c_void_p(stream)))
    assert err.value == 0
    assert np.array_equal(dev.cpu().numpy(), data)
