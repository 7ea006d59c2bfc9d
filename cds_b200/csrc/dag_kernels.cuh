// dag_kernels.cuh -- device code of the DAG orientation (see dag.cu).
#pragma once
#include "device_util.cuh"
#include "stages.h"

namespace {

using cds::HeavyBits;

__global__ void k_degree(const uint64_t *__restrict__ off, uint32_t n, uint32_t *__restrict__ deg) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    deg[v] = (uint32_t)(off[v + 1] - off[v]);
}

__device__ __forceinline__ bool above(uint32_t dw, uint32_t w, uint32_t dv, uint32_t v) {
  return dw > dv || (dw == dv && w > v);
}

// Warp per vertex, four groups of 32 neighbours in flight at a time: a hub's
// list is a chain of dependent loads (neighbour, then its degree), so this
// quarters the chain that bounds the kernel.
constexpr int DAG_U = 4;

__global__ void k_outdeg(const uint64_t *__restrict__ off, const uint32_t *__restrict__ adj,
                         const uint32_t *__restrict__ deg, uint32_t n,
                         uint32_t *__restrict__ outdeg, uint32_t *__restrict__ maxout) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  uint32_t local_max = 0;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
    const uint64_t b = off[v], e = off[v + 1];
    const uint32_t dv = (uint32_t)(e - b);
    uint32_t c = 0;
    for (uint64_t i0 = b + lane_id(); i0 < e; i0 += 32 * DAG_U) {
      uint32_t w[DAG_U];
#pragma unroll
      for (int u = 0; u < DAG_U; u++) w[u] = i0 + 32u * u < e ? adj[i0 + 32u * u] : 0xFFFFFFFFu;
#pragma unroll
      for (int u = 0; u < DAG_U; u++)
        if (w[u] != 0xFFFFFFFFu) c += above(deg[w[u]], w[u], dv, v);
    }
    c = warp_sum(c);
    if (lane_id() == 0) outdeg[v] = c;
    local_max = c > local_max ? c : local_max;
  }
  if (lane_id() == 0 && local_max) atomicMax(maxout, local_max);
}

// Heavy vertices: all of the graph, or the ones of largest degree.  Degrees are
// binned on a log scale, sixteen bins an octave, and the heavy ones are those
// from the lowest bin on at and above which at most `cap` vertices lie: a degree
// threshold, so that no DAG arc leaves the set.  Ids go by descending bin, so that the
// columns that the densest neighbourhoods touch lie together in every row.  bins[i] is
// left holding the next id of bin i, bins[512] the threshold bin.
constexpr uint32_t DEG_BINS = 512;
__device__ __forceinline__ uint32_t deg_bin(uint32_t d) {
  if (d < 16) return d;
  const uint32_t j = 31 - __clz(d);
  return 16 * (j - 3) + ((d >> (j - 4)) & 15u);
}
__global__ void k_deg_hist(const uint32_t *__restrict__ deg, uint32_t n, uint32_t *__restrict__ bins) {
  __shared__ uint32_t s[DEG_BINS];
  for (uint32_t i = threadIdx.x; i < DEG_BINS; i += blockDim.x) s[i] = 0;
  __syncthreads();
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    atomicAdd(&s[deg_bin(deg[v])], 1u);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < DEG_BINS; i += blockDim.x)
    if (s[i]) atomicAdd(&bins[i], s[i]);
}
__global__ void __launch_bounds__(DEG_BINS) k_heavy_bin(uint32_t *__restrict__ bins, uint32_t cap) {
  const uint32_t b = DEG_BINS - 1 - threadIdx.x;  // from the largest degree down
  uint32_t total;
  const uint32_t x = bins[b], above_b = block_exclusive_scan<uint32_t>(x, &total);
  const int ok = __syncthreads_count(above_b + x <= cap);  // a prefix of the threads
  bins[b] = above_b;
  if (threadIdx.x == 0) bins[DEG_BINS] = DEG_BINS - (uint32_t)ok;
}
__global__ void k_heavy_ids(const uint32_t *__restrict__ deg, uint32_t n, uint32_t *__restrict__ bins,
                            uint32_t *__restrict__ hid) {
  const uint32_t lo = bins[DEG_BINS];
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t b = deg_bin(deg[v]);
    hid[v] = b >= lo ? atomicAdd(&bins[b], 1u) : 0xFFFFFFFFu;
  }
}

// warp per vertex; writes the out-list in ascending id order plus padding, and
// both bits of an arc between heavy vertices
__global__ void k_dag_fill(const uint64_t *__restrict__ off, const uint32_t *__restrict__ adj,
                           const uint32_t *__restrict__ deg, uint32_t n,
                           const uint64_t *__restrict__ doff, uint32_t *__restrict__ dadj,
                           const HeavyBits hb, uint32_t *__restrict__ bits) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
    const uint64_t b = off[v], e = off[v + 1];
    const uint32_t dv = (uint32_t)(e - b);
    const uint32_t hv = hb.id(v);
    uint64_t w0 = doff[v];
    const uint64_t wend = doff[v + 1];
    for (uint64_t i0 = b; i0 < e; i0 += 32 * DAG_U) {
      uint32_t w[DAG_U];
      bool keep[DAG_U];
#pragma unroll
      for (int u = 0; u < DAG_U; u++) {
        const uint64_t i = i0 + 32u * u + lane_id();
        w[u] = i < e ? adj[i] : 0u;
      }
#pragma unroll
      for (int u = 0; u < DAG_U; u++) {
        const uint64_t i = i0 + 32u * u + lane_id();
        keep[u] = i < e && above(deg[w[u]], w[u], dv, v);
      }
      // groups in order, lanes in order within a group: ascending ids
#pragma unroll
      for (int u = 0; u < DAG_U; u++) {
        const uint32_t m = __ballot_sync(CDS_FULL, keep[u]);
        if (keep[u]) {
          dadj[w0 + __popc(m & ((1u << lane_id()) - 1u))] = w[u];
          if (hv != 0xFFFFFFFFu) {  // then w is heavy too
            const uint32_t hw = hb.id(w[u]);
            atomicOr(bits + (size_t)hv * hb.words + (hw >> 5), 1u << (hw & 31));
            atomicOr(bits + (size_t)hw * hb.words + (hv >> 5), 1u << (hv & 31));
          }
        }
        w0 += __popc(m);
      }
    }
    for (uint64_t i = w0 + lane_id(); i < wend; i += 32) dadj[i] = 0xFFFFFFFFu;
  }
}

}  // namespace
