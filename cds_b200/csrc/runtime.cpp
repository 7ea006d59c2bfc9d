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
// driver would keep.  At most MAX_BYTES a stream, and no more than the budget leaves
// beside what is in use; all of it goes back to the driver when it is in the way of an
// allocation and when the context ends.  The budget is checked against what is in use,
// as requested (the rounding adds at most a quarter of the small blocks to that).
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
size_t class_bytes(int size) {
  return size < 3 ? 256 * ((size_t)size + 1) : (size_t)(4 + (size - 3) % 4) << ((size - 3) / 4 + 8);
}

}  // namespace

void spare_release(cds_ctx *c) {
  for (auto &st : c->spare)
    for (int size = 0; size < SpareBlocks::SIZES; size++) {
      auto &v = st.second.blocks[size];
      for (void *p : v) cudaFreeAsync(p, st.first);
      c->held -= v.size() * class_bytes(size);
      st.second.bytes -= v.size() * class_bytes(size);
      v.clear();
    }
}

void *dalloc_bytes(cds_ctx *c, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return nullptr;
  bytes = (bytes + 255) & ~size_t(255);
  const uint64_t now = c->in_use.fetch_add(bytes) + bytes;
  void *p = nullptr;
  size_t held = 0;  // what the driver was asked for
  try {
    if (now > c->budget)
      fail(CDS_ERR_OOM, "device memory budget exceeded (" + std::to_string(now) + " > " +
                            std::to_string(c->budget) + " bytes)");
    {
      std::lock_guard<std::mutex> g(c->mu);
      size_t want = bytes;
      if (bytes <= SpareBlocks::MAX_BLOCK) {
        const int size = spare_size(bytes, &want);
        SpareBlocks &sp = c->spare[s];
        auto &v = sp.blocks[size];
        if (!v.empty()) {
          c->sizes[v.back()] = {bytes, want};
          p = v.back();
          v.pop_back();
          sp.bytes -= want;
        }
      }
      if (!p) {
        if (c->held + want > c->budget) spare_release(c);
        if (c->held + want > c->budget) want = bytes;
        c->held += held = want;
      }
    }
    if (!p) {
      cudaError_t e = cudaMallocFromPoolAsync(&p, held, c->pool, s);
      if (e != cudaSuccess) {
        cudaGetLastError();
        {
          std::lock_guard<std::mutex> g(c->mu);
          spare_release(c);
        }
        p = nullptr;
        e = cudaMallocFromPoolAsync(&p, held, c->pool, s);
      }
      if (e != cudaSuccess) {
        cudaGetLastError();
        p = nullptr;
        fail(CDS_ERR_OOM, std::string("device allocation failed: ") + cudaGetErrorString(e));
      }
      std::lock_guard<std::mutex> g(c->mu);
      c->sizes[p] = {bytes, held};
    }
  } catch (...) {
    if (held) {
      if (p) cudaFreeAsync(p, s);
      std::lock_guard<std::mutex> g(c->mu);
      c->held -= held;
    }
    c->in_use.fetch_sub(bytes);
    throw;
  }
  uint64_t pk = c->peak.load();
  while (now > pk && !c->peak.compare_exchange_weak(pk, now)) {
  }
  return p;
}

// Called by destructors: where keeping the block takes host memory that is not
// there, it goes back to the driver.
void dfree(cds_ctx *c, void *p, cudaStream_t s) {
  cds_ctx::Block b;
  bool kept = false;
  {
    std::lock_guard<std::mutex> g(c->mu);
    auto it = c->sizes.find(p);
    if (it != c->sizes.end()) {
      b = it->second;
      c->sizes.erase(it);
    }
    size_t rounded = 0;
    const int size = b.bytes && b.bytes <= SpareBlocks::MAX_BLOCK ? spare_size(b.bytes, &rounded) : -1;
    if (size >= 0 && b.held == rounded) try {
        SpareBlocks &sp = c->spare[s];
        if (sp.bytes + rounded <= SpareBlocks::MAX_BYTES) {
          sp.blocks[size].push_back(p);
          sp.bytes += rounded;
          kept = true;
        }
      } catch (const std::bad_alloc &) {
      }
    if (!kept) c->held -= b.held;
  }
  if (!kept) cudaFreeAsync(p, s);
  c->in_use.fetch_sub(b.bytes);
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
