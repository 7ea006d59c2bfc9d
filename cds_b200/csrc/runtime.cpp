// runtime.cpp -- what every stage stands on: errors, stream-ordered device memory
// against the context's budget, and reads back through pinned memory.  Host code
// only; no counterpart in the reference (cudaMalloc and pageable copies per stage).
#include <cstring>

#include "cds_internal.h"

namespace cds {

std::atomic<uint64_t> g_launches{0};

void fail(cds_status s, const std::string &msg) { throw Error{s, msg}; }

void cuda_check(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return;
  const cds_status s = (e == cudaErrorMemoryAllocation) ? CDS_ERR_OOM : CDS_ERR_CUDA;
  fail(s, std::string(what) + ": " + cudaGetErrorString(e));
}

// A solve makes about 60 allocations, most of them small, and the driver's calls for
// them were a tenth of the smallest solve's time (2,000 vertices: 0.91 -> 0.83 ms).
// Blocks of up to MAX_BLOCK bytes are therefore kept, by stream and rounded size, when
// they are freed: what a stream freed, its later work may use in the same order the
// driver would keep.  At most MAX_BYTES a stream; all of it goes back to the driver
// when an allocation fails and when the context ends.  The budget counts what is in
// use, as requested.
namespace {

// index and bytes of the rounded size (at most a quarter more than asked)
int spare_size(size_t bytes, size_t *rounded) {
  const uint64_t u = (bytes + 255) / 256;
  if (u < 4) {
    *rounded = u * 256;
    return (int)u - 1;
  }
  int e = 61 - __builtin_clzll(u);
  uint64_t q = (u + (1ull << e) - 1) >> e;
  if (q == 8) {
    q = 4;
    e++;
  }
  *rounded = (q << e) * 256;
  return 3 + 4 * e + (int)(q - 4);
}

}  // namespace

void spare_release(cds_ctx *c) {
  for (auto &st : c->spare) {
    for (auto &v : st.second.blocks) {
      for (void *p : v) cudaFreeAsync(p, st.first);
      v.clear();
    }
    st.second.bytes = 0;
  }
}

void *dalloc_bytes(cds_ctx *c, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return nullptr;
  bytes = (bytes + 255) & ~size_t(255);
  const uint64_t now = c->in_use.fetch_add(bytes) + bytes;
  if (now > c->budget) {
    c->in_use.fetch_sub(bytes);
    fail(CDS_ERR_OOM, "device memory budget exceeded (" + std::to_string(now) + " > " +
                          std::to_string(c->budget) + " bytes)");
  }
  const auto note_peak = [&] {
    uint64_t pk = c->peak.load();
    while (now > pk && !c->peak.compare_exchange_weak(pk, now)) {
    }
  };
  size_t rounded = bytes;
  void *p = nullptr;
  if (bytes <= SpareBlocks::MAX_BLOCK) {
    const int size = spare_size(bytes, &rounded);
    std::lock_guard<std::mutex> g(c->mu);
    SpareBlocks &sp = c->spare[s];
    if (!sp.blocks[size].empty()) {
      p = sp.blocks[size].back();
      sp.blocks[size].pop_back();
      sp.bytes -= rounded;
      c->sizes[p] = bytes;
      note_peak();
      return p;
    }
  }
  cudaError_t e = cudaMallocFromPoolAsync(&p, rounded, c->pool, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    {
      std::lock_guard<std::mutex> g(c->mu);
      spare_release(c);
    }
    e = cudaMallocFromPoolAsync(&p, rounded, c->pool, s);
  }
  if (e != cudaSuccess) {
    c->in_use.fetch_sub(bytes);
    cudaGetLastError();
    fail(CDS_ERR_OOM, std::string("device allocation failed: ") + cudaGetErrorString(e));
  }
  note_peak();
  std::lock_guard<std::mutex> g(c->mu);
  c->sizes[p] = bytes;
  return p;
}

void dfree(cds_ctx *c, void *p, cudaStream_t s) {
  size_t bytes = 0;
  bool kept = false;
  {
    std::lock_guard<std::mutex> g(c->mu);
    auto it = c->sizes.find(p);
    if (it != c->sizes.end()) {
      bytes = it->second;
      c->sizes.erase(it);
    }
    if (bytes && bytes <= SpareBlocks::MAX_BLOCK) {
      size_t rounded;
      const int size = spare_size(bytes, &rounded);
      SpareBlocks &sp = c->spare[s];
      if (sp.bytes + rounded <= SpareBlocks::MAX_BYTES) {
        sp.blocks[size].push_back(p);
        sp.bytes += rounded;
        kept = true;
      }
    }
  }
  if (!kept) cudaFreeAsync(p, s);
  c->in_use.fetch_sub(bytes);
}

namespace {
struct PinnedArea {
  char *p = nullptr;
  size_t cap = 0, top = 0;
  bool tried = false;
  ~PinnedArea() {
    if (p) (void)cudaFreeHost(p);  // at thread exit; an error here has no one to report to
  }
};
thread_local PinnedArea t_pinned;  // one per host thread, freed when the thread ends
constexpr size_t PINNED_BYTES = 1 << 20;
}  // namespace

HostReads::HostReads(cudaStream_t s) : s_(s), base_(t_pinned.top) {}

// (A stage that throws between add() and wait() leaves its copies queued: they land
// before the space is another group's, whose stream need not be theirs.)
HostReads::~HostReads() {
  for (const Item &it : items_)
    if (it.off != SIZE_MAX) {
      (void)cudaStreamSynchronize(s_);
      break;
    }
  t_pinned.top = base_;
}

void HostReads::add_bytes(void *dst, const void *src, size_t bytes) {
  if (!t_pinned.tried) {
    t_pinned.tried = true;
    if (cudaHostAlloc(reinterpret_cast<void **>(&t_pinned.p), PINNED_BYTES, cudaHostAllocPortable) ==
        cudaSuccess)
      t_pinned.cap = PINNED_BYTES;
    else
      (void)cudaGetLastError();  // no pinned memory: every read goes direct
  }
  const size_t off = (t_pinned.top + 15) & ~size_t(15);
  if (bytes && off + bytes <= t_pinned.cap) {
    items_.push_back({dst, src, off, bytes});
    t_pinned.top = off + bytes;
    CDS_CUDA(cudaMemcpyAsync(t_pinned.p + off, src, bytes, cudaMemcpyDeviceToHost, s_));
  } else {
    items_.push_back({dst, src, SIZE_MAX, bytes});
  }
}

void HostReads::wait() {
  for (const Item &it : items_)
    if (it.off == SIZE_MAX && it.bytes)
      CDS_CUDA(cudaMemcpyAsync(it.dst, it.src, it.bytes, cudaMemcpyDeviceToHost, s_));
  CDS_CUDA(cudaStreamSynchronize(s_));
  for (const Item &it : items_)
    if (it.off != SIZE_MAX) std::memcpy(it.dst, t_pinned.p + it.off, it.bytes);
  items_.clear();
  t_pinned.top = base_;
}

}  // namespace cds
