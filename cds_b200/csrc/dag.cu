// dag.cu -- orientation of the undirected CSR into a DAG.
//
// Replaces generateDAG (cudaCode/main.cu:22-57) with its kernels
// generateDegreeDAG / generateNeighborDAG (cudaCode/src/helpers.cu:112-173)
// and the host core ordering it depends on (cudaCode/src/graph.cpp:41-113).
// Each edge is oriented from the lower to the higher (degree, id) key, which
// bounds every out-degree by O(sqrt(m)) and needs no host-side ordering.  The
// k-clique set does not depend on the orientation.
//
// Out-lists keep ascending vertex ids and every row is padded to a multiple
// of 4 entries with 0xFFFFFFFF, so rows start on 16-byte boundaries and can
// be read with 128-bit loads.
#include "stages.h"
#include "device_util.cuh"

#include "dag_kernels.cuh"

#include <algorithm>

namespace cds {

namespace {

// The heavy vertices and their empty bitmap.  16,384 of them: 32 MB, which stays
// in L2 beside the lists; on R-MAT scale 18, edge factor 16, 99 % of the out-list
// entries a listing would search belong to them (8,192: 94 %; 32,768: 99.9 %).
// The bitmap takes at most an eighth of what the budget has left, as the stages to come
// need memory too (a small graph's needed 32 of 35 MB, and a budget of 34 refused what
// 2 MB hold): a context short of memory takes fewer, or none (every list is then
// searched).
constexpr uint32_t HEAVY_MAX = 16384, HEAVY_SHARE = 8;
void heavy_vertices(cds_ctx *c, cudaStream_t s, uint32_t n, Dag &dag) {
  dag.hid.c = dag.hbits.c = c;
  dag.hid.s = dag.hbits.s = s;
  const uint64_t used = c->in_use.load(), share = (c->budget > used ? c->budget - used : 0) / HEAVY_SHARE;
  for (uint32_t cap = std::min(n, HEAVY_MAX); cap >= 256 || cap == n; cap /= 2) {
    const uint32_t words = (cap + 31) / 32;
    if (4 * (uint64_t)cap * words > share) continue;
    try {
      dag.hbits.alloc((size_t)cap * words);
      if (cap < n) dag.hid.alloc(n);
    } catch (const Error &e) {
      if (e.status != CDS_ERR_OOM) throw;
      dag.hbits.release();
      continue;
    }
    dag.hbits.zero();
    dag.heavy.words = words;
    dag.heavy.bits = dag.hbits.p;
    if (cap < n) {
      DBuf<uint32_t> bins(c, s, DEG_BINS + 2);
      bins.zero();
      k_deg_hist<<<c->sm_count, 512, 0, s>>>(dag.deg.p, n, bins.p);
      k_heavy_bin<<<1, DEG_BINS, 0, s>>>(bins.p, cap);
      k_heavy_ids<<<c->sm_count * 4, 256, 0, s>>>(dag.deg.p, n, bins.p, dag.hid.p);
      count_launch(3);
      CDS_CUDA(cudaGetLastError());
      dag.heavy.hid = dag.hid.p;
    }
    return;
  }
}

}  // namespace

void build_dag(cds_ctx *c, cudaStream_t s, const uint64_t *off, const uint32_t *adj,
               uint32_t n, uint32_t k, Dag &dag) {
  dag.n = n;
  dag.deg.alloc(n + 1);
  dag.degree = dag.deg.p;
  dag.outdeg.alloc(n + 1);
  dag.off.alloc(n + 1);
  DBuf<uint32_t> maxout(c, s, 1);
  maxout.zero();
  if (n) {
    const int grid = c->sm_count * 8;
    k_degree<<<grid, 256, 0, s>>>(off, n, dag.deg.p);
    k_outdeg<<<grid, 256, 0, s>>>(off, adj, dag.deg.p, n, dag.outdeg.p, maxout.p);
    count_launch(2);
    CDS_CUDA(cudaGetLastError());
  }
  scan_u32_pad4(dag.outdeg.p, dag.off.p, n, c, s);
  uint64_t total = 0;
  {
    HostReads r(s);
    r.add(&total, dag.off.p + n);
    r.add(&dag.max_out, maxout.p);
    r.wait();
  }
  dag.adj.alloc(total + 4);
  if (n && k >= 3) heavy_vertices(c, s, n, dag);
  if (n) {
    k_dag_fill<<<c->sm_count * 8, 256, 0, s>>>(off, adj, dag.deg.p, n, dag.off.p, dag.adj.p, dag.heavy,
                                               dag.hbits.p);
    count_launch();
    CDS_CUDA(cudaGetLastError());
  }
}

}  // namespace cds
