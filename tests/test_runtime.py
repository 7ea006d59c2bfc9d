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
  const long left = news_left;  // (the test's own notes always fit)
  news_left = -1;
  live[*p] = n;
  news_left = left;
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


def test_kept_blocks_stay_within_the_budget(tmp_path):
    # sizes that are no other's class: what was kept for one does not serve the next
    run(tmp_path, """
      cds_ctx c;
      c.budget = 1 << 20;
      for (size_t n : {300u << 10, 200u << 10, 150u << 10, 700u << 10, 90u << 10, 1024u << 10}) {
        std::vector<void *> p;
        for (size_t i = 0; i < (1u << 20) / n; i++) p.push_back(dalloc_bytes(&c, n, stream(1 + i % 3)));
        for (size_t i = 0; i < p.size(); i++) dfree(&c, p[i], stream(1 + i % 3));
        assert(c.in_use.load() == 0);
      }
      assert(live_peak <= c.budget + c.budget / 4);  // (rounding, of blocks in use)
      assert(c.held == live_bytes);
    """)


def test_kept_blocks_serve_their_stream_and_are_bounded(tmp_path):
    run(tmp_path, """
      cds_ctx c;
      c.budget = 1ull << 40;
      void *a = dalloc_bytes(&c, 1000, stream(1));
      dfree(&c, a, stream(1));
      void *b = dalloc_bytes(&c, 1000, stream(2));
      assert(b != a && driver_calls == 2);
      assert(dalloc_bytes(&c, 900, stream(1)) == a && driver_calls == 2);
      dfree(&c, a, stream(1));
      dfree(&c, b, stream(2));
      std::vector<void *> p;
      for (int i = 0; i < 100; i++) p.push_back(dalloc_bytes(&c, 3u << 20, stream(1)));
      p.push_back(dalloc_bytes(&c, 64u << 20, stream(1)));
      for (void *q : p) dfree(&c, q, stream(1));
      assert(live_bytes <= SpareBlocks::MAX_BYTES + 1024);
      // an allocation that the driver refuses gets everything back first
      driver_limit = live_bytes + (1u << 20);
      void *d = dalloc_bytes(&c, 32u << 20, stream(2));
      assert(live_bytes == 32u << 20);
      dfree(&c, d, stream(2));
      bool refused = false;
      try {
        dalloc_bytes(&c, 1ull << 30, stream(2));
      } catch (const Error &e) {
        refused = e.status == CDS_ERR_OOM;
      }
      assert(refused && c.in_use.load() == 0 && live_bytes == 0);
    """)


def test_no_host_memory(tmp_path):
    # buffers are freed by destructors: a failure to keep a block must not leave them
    run(tmp_path, """
      for (long left = 0; left < 4; left++) {
        cds_ctx c;
        c.budget = 1ull << 40;
        std::vector<void *> p;
        for (int i = 0; i < 40; i++) p.push_back(dalloc_bytes(&c, 4096 << (i % 9), stream(1 + i % 2)));
        for (int i = 0; i < 40; i++) {
          news_left = left;
          dfree(&c, p[i], stream(3 + i % 5));
          news_left = -1;
        }
        assert(c.in_use.load() == 0);
        size_t before = live_bytes;
        int refused = 0;
        for (int i = 0; i < 8; i++) {
          news_left = i % 2 ? left : 0;
          try {
            void *q = dalloc_bytes(&c, 777777 + 4096 * i, stream(9));
            news_left = -1;
            dfree(&c, q, stream(9));
          } catch (...) {
            news_left = -1;
            refused++;
            assert(live_bytes == before);
          }
          before = live_bytes;
          assert(c.in_use.load() == 0);
        }
        assert(refused);
        spare_release(&c);
        assert(live_bytes == 0);
      }
    """)
