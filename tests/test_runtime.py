"""The runtime under the stages (device blocks kept by stream, reads back through
pinned memory), compiled by the host compiler against a CUDA runtime that the test
plays: copies that finish late, allocations that fail, host memory that runs out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

STUBS = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <new>
#include <vector>
#include "runtime.cpp"

struct Copy { void *dst; const void *src; size_t n; };
std::map<cudaStream_t, std::vector<Copy>> queued;      // copies a stream has not done yet
std::map<void *, size_t> live;                         // blocks the driver has given out
size_t live_bytes = 0, live_peak = 0, driver_limit = ~size_t(0), driver_calls = 0;
long news_left = -1;                                   // host allocations before one fails (-1: none does)

void run(cudaStream_t s) {
  for (const Copy &c : queued[s]) std::memcpy(c.dst, c.src, c.n);
  queued[s].clear();
}
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  queued[st].push_back({d, s, n});
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
  if (live_bytes + n > driver_limit) return cudaErrorMemoryAllocation;
  *p = std::malloc(1);
  live[*p] = n;
  live_bytes += n;
  if (live_bytes > live_peak) live_peak = live_bytes;
  driver_calls++;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
  assert(live.count(p));
  live_bytes -= live[p];
  live.erase(p);
  std::free(p);
  return cudaSuccess;
}
}
void *operator new(size_t n) {
  if (news_left == 0) throw std::bad_alloc();
  if (news_left > 0) news_left--;
  return std::malloc(n ? n : 1);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
cudaStream_t stream(long i) { return reinterpret_cast<cudaStream_t>(i); }
using namespace cds;
"""


def run(tmp_path, body):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(STUBS + "int main() {\n" + body + "\n}\n")
    subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "cds_b200", "csrc"), "-I", os.path.join(CUDA, "include"), "-o", str(exe),
                    str(src), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr


def test_reads_left_by_a_stage_that_throws(tmp_path):
    # a group is queued, its stage throws before the wait, and its stream runs late:
    # after the next group's copies and before that group takes its values
    run(tmp_path, """
      unsigned long long a = 7, b = 9, x = 0, y = 0;
      try {
        HostReads first(stream(1));
        first.add(&x, &a);
        fail(CDS_ERR_OOM, "the stage between");
      } catch (const Error &) {
      }
      HostReads second(stream(2));
      second.add(&y, &b);
      run(stream(2));
      run(stream(1));
      second.wait();
      assert(y == 9);
    """)


def test_nested_reads(tmp_path):
    run(tmp_path, """
      unsigned long long a = 1, b = 2, x = 0, y = 0;
      std::vector<char> big(2 << 20, 5), got(2 << 20, 0);
      HostReads outer(stream(1));
      outer.add(&x, &a);
      {
        HostReads inner(stream(1));
        inner.add(&y, &b);
        inner.add(got.data(), big.data(), big.size());  // past the pinned buffer: a direct copy
        inner.wait();
        assert(y == 2 && got == big);
      }
      outer.wait();
      assert(x == 1);
    """)
