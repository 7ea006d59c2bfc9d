// core.cu -- densest core, edge pruning, connected components, and the
// component-local clique/incidence layout the flow stage reads.
//
// Replaces generateDensestCore (cudaCode/main.cu:345-399, helpers.cu:821-896),
// prune (main.cu:400-449, helpers.cu:898-1041), componentDecompose
// (main.cu:451-518, helpers.cu:937-978) and the clique bucketing of
// getConnectedComponentStatus / rearrangeCliqueData (helpers.cu:1043-1096),
// and on the CPU side locateDensestCore, cliqueEnumerationListRecord,
// pruneInvalidEdges and connectedComponentDecompose
// (cpuCode/c++/src/helpers.cpp:710-1116).
//
//  - The (k',Psi)-core is every vertex with core number >= k' where
//    k' = ceil(best core density); its cliques are listed from the core's part
//    of the DAG (no other clique of the graph is ever written).
//  - Pruning marks each DAG arc covered by a core clique (clique records are
//    in orientation order, so member x -> member y is an arc for x < y).
//  - Components come from a lock-free union-find over the kept arcs (which
//    connect exactly what the core cliques connect) that always hangs the
//    larger root under the smaller one, so a component's root is its
//    smallest vertex and components are ordered as the reference's
//    ascending-start BFS orders them.
//  - Counters that many threads bump at once (per component, per instance)
//    are warp-aggregated: one atomic per distinct key in a warp.
#include "core_rows.cuh"
#include "device_util.cuh"
#include "stages.h"
#include "pipeline.h"

#include <algorithm>

namespace {

constexpr uint32_t NONE = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t inst_of(const uint32_t *of_vertex, uint32_t v) {
  return of_vertex ? of_vertex[v] : 0u;
}

// Grid-stride loops below step whole warps (base is warp-uniform), because
// the warp-aggregated atomics need all 32 lanes.
__global__ void k_core_flags(const uint32_t *__restrict__ core, const uint32_t *__restrict__ roots, uint32_t n,
                             const uint32_t *__restrict__ of_vertex,
                             const unsigned long long *__restrict__ kp, uint32_t *__restrict__ in_core,
                             unsigned long long *__restrict__ core_size,
                             unsigned long long *__restrict__ core_cliques) {
  for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t v = b + threadIdx.x;
    uint32_t i = 0, r = 0;
    bool in = false;
    if (v < n) {
      i = inst_of(of_vertex, v);
      const unsigned long long t = kp[i];
      in = t > 0 && (unsigned long long)core[v] >= t;
      in_core[v] = in;
      r = in ? roots[v] : 0u;  // a clique is in the core when its first member is
    }
    agg_add_u64(core_size, i, in);
    const uint32_t on = __ballot_sync(CDS_FULL, r != 0);
    if (!on) continue;
    const uint32_t i0 = __shfl_sync(CDS_FULL, i, __ffs(on) - 1);
    if (__all_sync(CDS_FULL, r == 0 || i == i0)) {
      const unsigned long long sum = warp_sum((unsigned long long)r);
      if (lane_id() == 0) atomicAdd(&core_cliques[i0], sum);
    } else if (r) {
      atomicAdd(&core_cliques[i], (unsigned long long)r);
    }
  }
}

// The core's part of the DAG: out-lists of core vertices, core neighbours only
// (ids as they are; other vertices get empty lists).  Warp per vertex, lists
// ascending and padded as the DAG's.
__global__ void k_core_outdeg(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                              const uint32_t *__restrict__ outdeg, const uint32_t *__restrict__ in_core, uint32_t n,
                              uint32_t *__restrict__ cout) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    uint32_t c = 0;
    if (in_core[u])
      for (uint32_t t = lane_id(); t < outdeg[u]; t += 32) c += in_core[dadj[doff[u] + t]];
    c = __reduce_add_sync(CDS_FULL, c);
    if (lane_id() == 0) cout[u] = c;
  }
}
__global__ void k_core_dag(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                           const uint32_t *__restrict__ outdeg, const uint32_t *__restrict__ in_core, uint32_t n,
                           const uint64_t *__restrict__ coff, uint32_t *__restrict__ cadj) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    if (!in_core[u]) continue;
    uint64_t at = coff[u];
    const uint64_t end = coff[u + 1];
    for (uint32_t t0 = 0; t0 < outdeg[u]; t0 += 32) {
      const uint32_t t = t0 + lane_id();
      const uint32_t w = t < outdeg[u] ? dadj[doff[u] + t] : 0u;
      const bool in = t < outdeg[u] && in_core[w];
      const uint32_t m = __ballot_sync(CDS_FULL, in);
      if (in) cadj[at + __popc(m & ((1u << lane_id()) - 1u))] = w;
      at += __popc(m);
    }
    for (uint64_t i = at + lane_id(); i < end; i += 32) cadj[i] = NONE;
  }
}
// arc u -> w of the DAG (w in the out-list of u), or NONE
__device__ __forceinline__ uint64_t find_arc(const uint64_t *doff, const uint32_t *dadj,
                                             const uint32_t *outdeg, uint32_t u, uint32_t w) {
  uint64_t lo = doff[u], hi = lo + outdeg[u];
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (dadj[mid] < w) lo = mid + 1;
    else hi = mid;
  }
  return (lo < doff[u] + outdeg[u] && dadj[lo] == w) ? lo : ~0ull;
}

__global__ void k_mark_arcs(const uint32_t *__restrict__ members, uint64_t m, uint32_t k,
                            const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                            const uint32_t *__restrict__ outdeg,
                            uint8_t *__restrict__ arc_keep, uint32_t *__restrict__ err) {
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t *r = members + c * k;
    for (uint32_t x = 0; x < k; x++)
      for (uint32_t y = x + 1; y < k; y++) {
        const uint64_t a = find_arc(doff, dadj, outdeg, r[x], r[y]);
        if (a == ~0ull) atomicOr(err, DEV_ERR_INTERNAL);
        else arc_keep[a] = 1;
      }
  }
}

// Small cores (every instance's at most PAIR_CORE_MAX vertices, its bitmaps together
// within the budget's share): adjacency and the pairs that core cliques cover are
// bitmaps over core-local ids, an instance's rows as wide as its own core (24 graphs
// in four batches, cores of 5,786 vertices in the largest: 66 -> 34 ms, where
// rows over all ids left that batch to listing and flows).  For k <= 5 a pair is
// tested on the adjacency rows alone (does a clique of the k-2 other members fit
// into the common neighbours?), which in a dense core the first candidate answers;
// for larger k the listed cliques mark their pairs.  An edge covers itself, so k = 2
// needs no such test and takes larger cores.
constexpr uint32_t PAIR_CORE_MAX = 4096, EDGE_CORE_MAX = 16384;
constexpr uint64_t BAND_BYTES = 4ull << 20;  // of both bitmaps, whatever the budget

__global__ void k_core_bits(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                            const uint32_t *__restrict__ outdeg, const uint32_t *__restrict__ in_core,
                            const uint64_t *__restrict__ lid, const uint32_t *__restrict__ core_vertex,
                            uint32_t ncore, CoreRows r, uint32_t *__restrict__ adj) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < ncore; i += warps) {
    const uint32_t u = core_vertex[i], d = outdeg[u];
    const CoreBand bd = band_of(r, u);
    uint32_t *rows = adj + bd.word;
    const uint32_t a = i - bd.lid;
    for (uint32_t t = lane_id(); t < d; t += 32) {
      const uint32_t w = dadj[doff[u] + t];
      if (!in_core[w]) continue;
      const uint32_t b = (uint32_t)lid[w] - bd.lid;
      atomicOr(rows + a * bd.width + (b >> 5), 1u << (b & 31));
      atomicOr(rows + b * bd.width + (a >> 5), 1u << (a & 31));
    }
  }
}

// is there a D-clique among the vertices of mask M (words lane, lane + 32, ...)?
template <int D>
__device__ bool clique_in(const uint32_t (&M)[PAIR_CORE_MAX / 1024], const uint32_t *adj, uint32_t words) {
  constexpr uint32_t Q = PAIR_CORE_MAX / 1024;
  if constexpr (D == 0) {
    return true;
  } else if constexpr (D == 1) {
    uint32_t any = 0;
#pragma unroll
    for (uint32_t q = 0; q < Q; q++) any |= M[q];
    return __any_sync(CDS_FULL, any != 0);
  } else {
#pragma unroll
    for (uint32_t q = 0; q < Q; q++)
      for (uint32_t on = __ballot_sync(CDS_FULL, M[q] != 0); on; on &= on - 1) {
        const uint32_t l = __ffs(on) - 1;
        for (uint32_t m = __shfl_sync(CDS_FULL, M[q], l); m; m &= m - 1) {
          const uint32_t j = (q * 32 + l) * 32 + __ffs(m) - 1;
          uint32_t N[Q];
#pragma unroll
          for (uint32_t x = 0; x < Q; x++) {
            const uint32_t w = x * 32 + lane_id();
            N[x] = w < words ? M[x] & adj[(size_t)j * words + w] : 0u;
          }
          if (clique_in<D - 1>(N, adj, words)) return true;
        }
      }
    return false;
  }
}

// bits: the covered pairs a < b; pairs counted per instance.  Warp per row word.
// (bits comes in zeroed.)  parent: each id's smallest partner below it, which leaves
// the union-find over the pairs little to join.
template <int K>
__global__ void k_cover(const uint32_t *__restrict__ all, CoreRows r, uint32_t ncore,
                        const uint32_t *__restrict__ core_vertex, uint32_t *__restrict__ bits,
                        uint32_t *parent, unsigned long long *__restrict__ pairs) {
  constexpr uint32_t Q = PAIR_CORE_MAX / 1024;
  each_word(r, ncore, core_vertex, all, [&](uint32_t i, const CoreBand &bd, uint32_t w0, uint32_t m) {
    const uint32_t *adj = all + bd.word;
    const uint32_t a = i - bd.lid, words = bd.width;
    uint32_t out = 0;
    if (w0 == (a >> 5)) m &= ~((2u << (a & 31)) - 1u);
    if (K == 2) out = m;
    for (uint32_t rest = K == 2 ? 0u : m; rest; rest &= rest - 1) {
      const uint32_t b = w0 * 32 + __ffs(rest) - 1;
      uint32_t M[Q];
#pragma unroll
      for (uint32_t q = 0; q < Q; q++) {
        const uint32_t w = q * 32 + lane_id();
        M[q] = w < words ? adj[(size_t)a * words + w] & adj[(size_t)b * words + w] : 0u;
      }
      if (clique_in<K - 2>(M, adj, words)) out |= rest & (0u - rest);
    }
    const uint32_t b = bd.lid + w0 * 32 + lane_id();
    if (((out >> lane_id()) & 1u) && __ldcg(parent + b) > i) atomicMin(parent + b, i);
    if (lane_id() == 0 && out) {
      bits[bd.word + a * words + w0] = out;
      atomicAdd(&pairs[inst_of(r.of_vertex, core_vertex[i])], (unsigned long long)__popc(out));
    }
  });
}

// core-local ids in vertex order: in_core scanned into lid, and the inverse
// core_vertex[lid] = v (so the smallest id of a set of core vertices is its
// smallest vertex)
__global__ void k_core_vertex(const uint32_t *__restrict__ in_core, const uint64_t *__restrict__ lid, uint32_t n,
                              uint32_t *__restrict__ core_vertex, uint32_t *__restrict__ parent) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    if (in_core[v]) {
      const uint32_t a = (uint32_t)lid[v];
      core_vertex[a] = v;
      parent[a] = a;
    }
}

// k >= 6.  Bits are of pairs a < b, as k_cover's: a record's members are in the order
// of the DAG, which climbs in degree and not in id.
__global__ void k_mark_pairs(const uint32_t *__restrict__ members, uint64_t m, uint32_t k,
                             const uint64_t *__restrict__ lid, CoreRows rows, uint32_t *__restrict__ all) {
  for (uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m;
       c += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t *r = members + c * k;
    const CoreBand bd = band_of(rows, r[0]);
    for (uint32_t x = 0; x < k; x++) {
      const uint32_t u = (uint32_t)lid[r[x]] - bd.lid;
      for (uint32_t y = x + 1; y < k; y++) {
        const uint32_t v = (uint32_t)lid[r[y]] - bd.lid, a = min(u, v), b = max(u, v);
        uint32_t *w = all + bd.word + a * bd.width + (b >> 5);
        const uint32_t bit = 1u << (b & 31);
        if (!(*(volatile uint32_t *)w & bit)) atomicOr(w, bit);
      }
    }
  }
}

__global__ void k_pairs_to_arcs(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                                const uint32_t *__restrict__ outdeg, const uint32_t *__restrict__ in_core,
                                const uint64_t *__restrict__ lid, uint32_t n, CoreRows rows,
                                const uint32_t *__restrict__ bits, uint8_t *__restrict__ arc_keep) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    if (!in_core[u]) continue;
    const CoreBand bd = band_of(rows, u);
    const uint32_t a = (uint32_t)lid[u] - bd.lid;
    for (uint32_t t = lane_id(); t < outdeg[u]; t += 32) {
      const uint32_t w = dadj[doff[u] + t];
      if (!in_core[w]) continue;
      const uint32_t b = (uint32_t)lid[w] - bd.lid, lo = min(a, b), hi = max(a, b);
      if (bits[bd.word + lo * bd.width + (hi >> 5)] & (1u << (hi & 31))) arc_keep[doff[u] + t] = 1;
    }
  }
}

// warp per vertex: kept arcs per instance
__global__ void k_count_arcs(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ outdeg,
                             const uint8_t *__restrict__ arc_keep, uint32_t n,
                             const uint32_t *__restrict__ of_vertex,
                             unsigned long long *__restrict__ out) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
    uint32_t c = 0;
    for (uint32_t t = lane_id(); t < outdeg[v]; t += 32) c += arc_keep[doff[v] + t];
    c = warp_sum(c);
    if (lane_id() == 0 && c) atomicAdd(&out[inst_of(of_vertex, v)], (unsigned long long)c);
  }
}

__device__ __forceinline__ uint32_t uf_find(uint32_t *parent, uint32_t x) {
  uint32_t p = parent[x];
  while (p != x) {
    const uint32_t gp = parent[p];
    if (gp != p) parent[x] = gp;  // path halving; only ever points closer to the root
    x = p;
    p = gp;
  }
  return x;
}

__device__ __forceinline__ void unite(uint32_t *parent, uint32_t a, uint32_t b, uint32_t *err) {
  for (int tries = 0;; tries++) {
    if (tries > (1 << 20)) {
      atomicOr(err, DEV_ERR_TIMEOUT);
      return;
    }
    const uint32_t ra = uf_find(parent, a), rb = uf_find(parent, b);
    if (ra == rb) return;
    const uint32_t lo = ra < rb ? ra : rb, hi = ra < rb ? rb : ra;
    if (atomicCAS(&parent[hi], hi, lo) == hi) return;
    a = lo;
    b = hi;
  }
}

// of a small core: union-find over the covered pairs of the bitmap, by core-local id
// (a warp a word: one block over all of them took 62 us at 463 vertices, with its two launches; this 50)
__global__ void k_union_bits(const uint32_t *__restrict__ bits, CoreRows r, uint32_t ncore,
                             const uint32_t *__restrict__ core_vertex, uint32_t *parent, uint32_t *err) {
  each_word(r, ncore, core_vertex, bits, [&](uint32_t a, const CoreBand &bd, uint32_t w, uint32_t m) {
    if (!((m >> lane_id()) & 1u)) return;
    const uint32_t b = bd.lid + w * 32 + lane_id();
    if (__ldcg(parent + a) != __ldcg(parent + b)) unite(parent, a, b, err);
  });
}
__global__ void k_roots_bits(uint32_t *parent, const uint32_t *__restrict__ in_core, const uint64_t *__restrict__ lid,
                             const uint32_t *__restrict__ core_vertex, uint32_t n, uint32_t *__restrict__ comp) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    comp[v] = in_core[v] ? core_vertex[uf_find(parent, (uint32_t)lid[v])] : NONE;
}

// union-find over the kept arcs: they connect exactly what the core cliques
// connect, with at most m unions instead of (k-1)|Psi|
__global__ void k_union(const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                        const uint32_t *__restrict__ outdeg, const uint8_t *__restrict__ keep,
                        uint32_t n, uint32_t *parent, uint32_t *err) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    for (uint32_t t = lane_id(); t < outdeg[u]; t += 32) {
      if (!keep[doff[u] + t]) continue;
      unite(parent, u, dadj[doff[u] + t], err);
    }
  }
}

__global__ void k_roots(uint32_t *parent, const uint32_t *__restrict__ in_core, uint32_t n,
                        uint32_t *__restrict__ comp) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    comp[v] = in_core[v] ? uf_find(parent, v) : NONE;
}

// Core cliques per component: every core clique lies in its first member's.
__global__ void k_comp_cliques(const uint32_t *__restrict__ roots, uint32_t n, const uint32_t *__restrict__ comp,
                               unsigned long long *__restrict__ ccount) {
  for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t u = b + threadIdx.x;
    const uint32_t r = u < n ? comp[u] : NONE;
    const unsigned long long c = r != NONE ? roots[u] : 0ull;
    const uint32_t on = __ballot_sync(CDS_FULL, c != 0);
    if (!on) continue;
    const uint32_t r0 = __shfl_sync(CDS_FULL, r, __ffs(on) - 1);
    if (__all_sync(CDS_FULL, c == 0 || r == r0)) {  // one component in the warp, mostly
      const unsigned long long sum = warp_sum(c);
      if (lane_id() == 0) atomicAdd(&ccount[r0], sum);
    } else if (c) {
      atomicAdd(&ccount[r], c);
    }
  }
}

// roots of components with >= 1 clique; component counts per instance
__global__ void k_root_flags(const uint32_t *__restrict__ comp, const unsigned long long *__restrict__ ccount,
                             uint32_t n, const uint32_t *__restrict__ of_vertex,
                             uint32_t *__restrict__ is_root, unsigned long long *__restrict__ ncomp) {
  for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t v = b + threadIdx.x;
    bool root = false;
    if (v < n) {
      root = comp[v] == v;
      is_root[v] = root && ccount[v] > 0;
    }
    agg_add_u64(ncomp, root ? inst_of(of_vertex, v) : 0u, root);
  }
}

__global__ void k_comp_sizes(const uint32_t *__restrict__ comp, const uint64_t *__restrict__ cidx,
                             const unsigned long long *__restrict__ ccount, uint32_t n,
                             uint32_t *__restrict__ csize, unsigned long long *__restrict__ cclq,
                             const uint32_t *__restrict__ core, uint32_t *__restrict__ cmax) {
  for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t v = b + threadIdx.x;
    bool in = false;
    uint32_t ci = 0;
    if (v < n) {
      const uint32_t r = comp[v];
      in = r != NONE && ccount[r] > 0;
      if (in) {
        ci = (uint32_t)cidx[r];
        if (r == v) cclq[ci] = ccount[r];
      }
    }
    agg_inc(csize, ci, in);
    const uint32_t grp = __match_any_sync(CDS_FULL, in ? ci : NONE);
    const uint32_t mx = __reduce_max_sync(grp, in ? core[v] : 0u);
    if (in && (int)lane_id() == __ffs(grp) - 1) atomicMax(&cmax[ci], mx);
  }
}

__global__ void k_local_ids(const uint32_t *__restrict__ comp, const uint64_t *__restrict__ cidx,
                            const unsigned long long *__restrict__ ccount, uint32_t n,
                            const uint64_t *__restrict__ vbeg, uint32_t *__restrict__ vcur,
                            uint32_t *__restrict__ local, uint32_t *__restrict__ vmap,
                            uint32_t *__restrict__ vcnet) {
  for (uint32_t b = blockIdx.x * blockDim.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t v = b + threadIdx.x;
    bool in = false;
    uint32_t ci = 0;
    if (v < n) {
      const uint32_t r = comp[v];
      in = r != NONE && ccount[r] > 0;
      if (in) ci = (uint32_t)cidx[r];
      else local[v] = NONE;
    }
    const uint32_t slot = agg_inc(vcur, ci, in);
    if (in) {
      const uint32_t l = (uint32_t)vbeg[ci] + slot;
      local[v] = l;
      vmap[l] = v;
      vcnet[l] = ci;
    }
  }
}

// Networks of at most this many vertices (all components of a problem
// together) count per-vertex degrees and cursors per block in shared memory.
constexpr uint32_t SMALL_NV = 2048;

// Core cliques grouped by component, in the local ids of their networks.
// A block whose core cliques all lie in one component (the usual case) takes
// its slots with one atomic; otherwise each warp takes its own.
__global__ void k_bucket_cliques(const uint32_t *__restrict__ members, uint64_t m, uint32_t k,
                                 const uint32_t *__restrict__ comp, const uint64_t *__restrict__ cidx,
                                 const uint8_t *__restrict__ open, const uint64_t *__restrict__ cbeg,
                                 unsigned long long *__restrict__ ccur, const uint32_t *__restrict__ local,
                                 uint32_t nv, uint32_t *__restrict__ rec, uint32_t *__restrict__ ldeg) {
  __shared__ uint32_t s_lo, s_hi;
  __shared__ unsigned long long s_base;
  __shared__ uint32_t s_ldeg[SMALL_NV];  // this block's degree counts (nv <= SMALL_NV)
  const bool small = nv <= SMALL_NV;
  if (small) {
    for (uint32_t l = threadIdx.x; l < nv; l += blockDim.x) s_ldeg[l] = 0;
    __syncthreads();
  }
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < m; b += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t c = b + threadIdx.x;
    bool in = c < m;
    const uint32_t *r = members + (in ? c : 0) * k;
    const uint32_t ci = in ? (uint32_t)cidx[comp[r[0]]] : 0u;
    in = in && open[ci];
    if (threadIdx.x == 0) {
      s_lo = 0xFFFFFFFFu;
      s_hi = 0;
    }
    __syncthreads();
    const uint32_t lo = warp_min(in ? ci : 0xFFFFFFFFu), hi = warp_max(in ? ci : 0u);
    if (lane_id() == 0) {
      atomicMin(&s_lo, lo);
      atomicMax(&s_hi, hi);
    }
    __syncthreads();
    unsigned long long slot;
    if (s_lo == s_hi) {  // one component in the block (s_lo > s_hi: none)
      uint32_t total;
      const uint32_t rank = block_exclusive_scan<uint32_t>(in ? 1u : 0u, &total);
      if (threadIdx.x == 0) s_base = atomicAdd(&ccur[s_lo], (unsigned long long)total);
      __syncthreads();
      slot = s_base + rank;
    } else {
      slot = agg_inc_u64(ccur, ci, in);
    }
    const uint64_t pos = in ? cbeg[ci] + slot : 0;
    // the rest of the record (spare slots, flow words) starts at zero, so
    // the first flow over these records needs no reset pass
    if (k <= 4) {
      // the whole record in 16-byte stores (one for k = 2, two for k = 3, 4)
      uint32_t l[4] = {0u, 0u, 0u, 0u};
      if (k == 4 && in) {
        const uint4 q = *reinterpret_cast<const uint4 *>(members + c * 4);
        l[0] = local[q.x];
        l[1] = local[q.y];
        l[2] = local[q.z];
        l[3] = local[q.w];
      } else if (in) {
        for (uint32_t j = 0; j < k; j++) l[j] = local[r[j]];
      }
#pragma unroll
      for (uint32_t j = 0; j < 4; j++)
        if (j < k) agg_add_u32(small ? s_ldeg : ldeg, l[j], in);
      if (in) {
        uint4 *R = reinterpret_cast<uint4 *>(rec + (pos << rec_shift(k)));
        R[0] = make_uint4(l[0], l[1], l[2], l[3]);
        if (k > 2) R[1] = make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
      for (uint32_t j = 0; j < k; j++) {
        const uint32_t l = in ? local[r[j]] : 0u;
        if (in) rec[(pos << rec_shift(k)) + j] = l;
        agg_add_u32(small ? s_ldeg : ldeg, l, in);
      }
      if (in)
        for (uint32_t j = k; j < 2 * rec_slots(k); j++) rec[(pos << rec_shift(k)) + j] = 0u;
    }
    __syncthreads();  // s_lo, s_hi and s_base are reused by the next tile
  }
  if (small)
    for (uint32_t l = threadIdx.x; l < nv; l += blockDim.x)
      if (s_ldeg[l]) atomicAdd(&ldeg[l], s_ldeg[l]);
}

template <typename I>
__global__ void k_fill_vinc(const uint32_t *__restrict__ rec, uint64_t nc, uint32_t k,
                            const uint64_t *__restrict__ vinc_off, uint32_t *__restrict__ cur,
                            I *__restrict__ vinc) {
  // slot-major walk (slot j of every clique, then slot j+1): lanes see the
  // same slot of consecutive cliques, which often share that member, so the
  // cursor atomics aggregate
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint32_t j = 0; j < k; j++) {
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < nc; b += stride) {
      const uint64_t c = b + threadIdx.x;
      const bool in = c < nc;
      const uint32_t l = in ? rec[(c << rec_shift(k)) + j] : 0u;
      const uint32_t slot = agg_inc(cur, l, in);
      if (in) vinc[vinc_off[l] + slot] = (I)c;
    }
  }
}

// The same for networks of at most SMALL_NV vertices, where the per-vertex
// cursors would be a few hundred hot words: each block takes a contiguous
// range of cliques, counts its incidences per vertex in shared memory,
// reserves one range per vertex with a single atomic, then writes.
template <typename I>
__global__ void k_fill_vinc_small(const uint32_t *__restrict__ rec, uint64_t nc, uint32_t k, uint32_t nv,
                                  const uint64_t *__restrict__ vinc_off, uint32_t *__restrict__ cur,
                                  I *__restrict__ vinc) {
  __shared__ uint32_t s_cnt[SMALL_NV], s_base[SMALL_NV];
  const uint64_t per = (nc + gridDim.x - 1) / gridDim.x;
  const uint64_t c_lo = min(nc, (uint64_t)blockIdx.x * per), c_hi = min(nc, c_lo + per);
  for (uint32_t l = threadIdx.x; l < nv; l += blockDim.x) s_cnt[l] = 0;
  __syncthreads();
  // a thread per clique record (consecutive threads, consecutive records,
  // which share their first members: lanes in runs of one member reserve
  // together, not 32 conflicting atomics on one word)
  const uint32_t rs = rec_shift(k);
  for (uint64_t c0 = c_lo; c0 < c_hi; c0 += blockDim.x) {
    const uint64_t c = c0 + threadIdx.x;
    const bool in = c < c_hi;
    for (uint32_t j = 0; j < k; j++) run_inc(s_cnt, in ? rec[(c << rs) + j] : 0u, in);
  }
  __syncthreads();
  for (uint32_t l = threadIdx.x; l < nv; l += blockDim.x) {
    const uint32_t n_l = s_cnt[l];
    s_base[l] = n_l ? atomicAdd(&cur[l], n_l) : 0u;
    s_cnt[l] = 0;
  }
  __syncthreads();
  for (uint64_t c0 = c_lo; c0 < c_hi; c0 += blockDim.x) {
    const uint64_t c = c0 + threadIdx.x;
    const bool in = c < c_hi;
    for (uint32_t j = 0; j < k; j++) {
      const uint32_t l = in ? rec[(c << rs) + j] : 0u;
      const uint32_t at = run_inc(s_cnt, l, in);
      if (in) vinc[vinc_off[l] + s_base[l] + at] = (I)c;
    }
  }
}

__global__ void k_iota(uint32_t *__restrict__ a, uint32_t n) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) a[v] = v;
}

__global__ void k_gather_roots(const uint32_t *__restrict__ is_root, const uint64_t *__restrict__ cidx,
                               uint32_t n, uint32_t *__restrict__ roots) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    if (is_root[v]) roots[cidx[v]] = v;
}

}  // namespace

namespace cds {

namespace {

// Every clique of the densest core, from the core's part of the DAG.
void list_core_cliques(cds_ctx *c, cudaStream_t s, const Dag &gdag, uint32_t k, const Tuning &t, CoreOut &out,
                       Dag &dag, const CountHook *on_count) {
  const uint32_t n = gdag.n;
  const int G = c->sm_count * 8;
  dag.n = n;
  dag.max_out = gdag.max_out;
  dag.heavy = gdag.heavy;
  dag.degree = gdag.degree;
  dag.outdeg = DBuf<uint32_t>(c, s, n + 1);
  dag.off = DBuf<uint64_t>(c, s, n + 1);
  dag.adj = DBuf<uint32_t>(c, s, gdag.adj.n);
  {
    ProfScope ps(c, s, "core_dag");
    if (n)
      k_core_outdeg<<<G, 256, 0, s>>>(gdag.off.p, gdag.adj.p, gdag.outdeg.p, out.in_core.p, n, dag.outdeg.p);
    scan_u32_pad4(dag.outdeg.p, dag.off.p, n, c, s);
    if (n)
      k_core_dag<<<G, 256, 0, s>>>(gdag.off.p, gdag.adj.p, gdag.outdeg.p, out.in_core.p, n, dag.off.p, dag.adj.p);
    count_launch(2);
    CDS_CUDA(cudaGetLastError());
  }
  list_cliques(c, s, dag, k, LIST_WRITE, t, out.cliques, on_count);
  out.listed = true;
}

}  // namespace

void densest_core_and_components(cds_ctx *c, cudaStream_t s, const Dag &gdag, const PeelOut &pe,
                                 const Instances &inst, uint32_t k, const Tuning &t, CoreOut &out,
                                 StageClock *clk, const CountHook *on_count) {
  const uint32_t n = gdag.n;
  const uint32_t ninst = inst.count;
  const uint32_t *of_vertex = ninst > 1 ? inst.of_vertex.p : nullptr;
  const int G = c->sm_count * 8;

  out.threshold.assign(ninst, 0);
  for (uint32_t i = 0; i < ninst; i++)
    if (pe.best_den[i] && pe.best_num[i])
      out.threshold[i] = (pe.best_num[i] + pe.best_den[i] - 1) / pe.best_den[i];
  DBuf<unsigned long long> kp(c, s, ninst);
  CDS_CUDA(cudaMemcpyAsync(kp.p, out.threshold.data(), ninst * 8, cudaMemcpyHostToDevice, s));
  DBuf<unsigned long long> stats(c, s, 4 * (size_t)ninst);  // core size, core cliques, pairs, comps
  stats.zero();
  DBuf<uint32_t> err(c, s, 1);
  err.zero();
  out.in_core = DBuf<uint32_t>(c, s, n + 1);
  const DBuf<uint32_t> &in_core = out.in_core;
  if (n) {
    ProfScope ps(c, s, "core_flags");
    k_core_flags<<<G, 256, 0, s>>>(pe.core.p, pe.roots.p, n, of_vertex, kp.p, in_core.p, stats.p, stats.p + ninst);
    count_launch();
    CDS_CUDA(cudaGetLastError());
  }
  if (clk) out.mk_core = clk->mark();

  // prune: pairs inside >= 1 core clique
  uint64_t ncore = 0, m = 0;
  std::vector<unsigned long long> hstats(2 * (size_t)ninst);
  {
    HostReads r(s);
    r.add(hstats.data(), stats.p, hstats.size());
    r.wait();
    for (uint32_t i = 0; i < ninst; i++) {
      ncore += hstats[i];
      m += hstats[ninst + i];
    }
  }
  // marks over core-local ids; k <= 5: ... found on the adjacency alone
  bool bitmap = m && n;
  uint64_t words = 0;  // of a bitmap
  {
    std::vector<CoreBand> band(ninst);
    uint64_t at = 0;
    for (uint32_t i = 0; i < ninst; i++) {
      const uint64_t size = hstats[i], width = (size + 31) / 32;
      if (size > (k == 2 ? EDGE_CORE_MAX : PAIR_CORE_MAX)) bitmap = false;
      band[i] = CoreBand{(uint32_t)at, (uint32_t)width, (uint32_t)words};
      at += size;
      words += size * width;
      out.rows.words = std::max(out.rows.words, (uint32_t)width);
      if (8 * words > std::max<uint64_t>(BAND_BYTES, c->budget / 64)) bitmap = false;
    }
    if (bitmap) {
      out.band = DBuf<CoreBand>(c, s, ninst);
      CDS_CUDA(cudaMemcpyAsync(out.band.p, band.data(), ninst * sizeof(CoreBand), cudaMemcpyHostToDevice, s));
      out.rows.of_vertex = of_vertex;
      out.rows.band = out.band.p;
    }
  }
  out.small = bitmap && k <= 5;
  out.ncore = (uint32_t)ncore;
  DBuf<uint64_t> lid(c, s, bitmap ? n + 1 : 0);
  DBuf<uint8_t> keep(c, s, 0);
  DBuf<uint32_t> parent(c, s, bitmap ? ncore + 1 : n + 1);  // union-find, of core-local ids or vertices
  Dag dag;  // of the core, when its cliques are listed
  if (m && !out.small) list_core_cliques(c, s, gdag, k, t, out, dag, on_count);
  {
    ProfScope ps(c, s, "prune_arcs");
    if (bitmap) {
      out.core_vertex = DBuf<uint32_t>(c, s, ncore + 1);
      out.bits = DBuf<uint32_t>(c, s, words + 1);
      out.bits.zero();
      scan_u32(in_core.p, lid.p, n, c, s);
      k_core_vertex<<<G, 256, 0, s>>>(in_core.p, lid.p, n, out.core_vertex.p, parent.p);
      count_launch();
    }
    if (out.small) {
      DBuf<uint32_t> adj(c, s, words + 1);
      adj.zero();
      k_core_bits<<<G, 256, 0, s>>>(gdag.off.p, gdag.adj.p, gdag.outdeg.p, in_core.p, lid.p, out.core_vertex.p,
                                    (uint32_t)ncore, out.rows, adj.p);
      void (*cover)(const uint32_t *, CoreRows, uint32_t, const uint32_t *, uint32_t *, uint32_t *,
                    unsigned long long *) =
           k == 2 ? k_cover<2> : k == 3 ? k_cover<3> : k == 4 ? k_cover<4> : k_cover<5>;
      cover<<<G, 256, 0, s>>>(adj.p, out.rows, (uint32_t)ncore, out.core_vertex.p, out.bits.p, parent.p,
                              stats.p + 2 * ninst);
      count_launch(2);
    } else if (m) {
      keep.alloc(dag.adj.n + 1);
      keep.zero();
      const Cliques &cl = out.cliques;
      if (bitmap) {
        k_mark_pairs<<<G, 256, 0, s>>>(cl.members.p, m, k, lid.p, out.rows, out.bits.p);
        k_pairs_to_arcs<<<G, 256, 0, s>>>(dag.off.p, dag.adj.p, dag.outdeg.p, in_core.p, lid.p, n, out.rows, out.bits.p,
                                          keep.p);
        count_launch();
      } else {
        k_mark_arcs<<<G, 256, 0, s>>>(cl.members.p, m, k, dag.off.p, dag.adj.p, dag.outdeg.p, keep.p, err.p);
      }
      k_count_arcs<<<G, 256, 0, s>>>(dag.off.p, dag.outdeg.p, keep.p, n, of_vertex, stats.p + 2 * ninst);
      count_launch(2);
    }
    CDS_CUDA(cudaGetLastError());
  }
  if (clk) out.mk_prune = clk->mark();

  // components
  out.comp = DBuf<uint32_t>(c, s, n + 1);
  out.cidx = DBuf<uint64_t>(c, s, n + 1);
  const DBuf<uint32_t> &comp = out.comp;
  const DBuf<uint64_t> &cidx = out.cidx;
  DBuf<uint32_t> is_root(c, s, n + 1);
  DBuf<unsigned long long> ccount(c, s, n + 1);  // core cliques per component root (may pass 2^32)
  ccount.zero();
  {
    ProfScope ps_cc(c, s, "components_unionfind");
    if (bitmap) {
      k_union_bits<<<G, 256, 0, s>>>(out.bits.p, out.rows, (uint32_t)ncore, out.core_vertex.p, parent.p, err.p);
      k_roots_bits<<<G, 256, 0, s>>>(parent.p, in_core.p, lid.p, out.core_vertex.p, n, comp.p);
      count_launch(2);
    } else if (n) {
      k_iota<<<G, 256, 0, s>>>(parent.p, n);
      if (m) k_union<<<G, 256, 0, s>>>(dag.off.p, dag.adj.p, dag.outdeg.p, keep.p, n, parent.p, err.p);
      k_roots<<<G, 256, 0, s>>>(parent.p, in_core.p, n, comp.p);
      count_launch(3);
    }
    if (n) {
      k_comp_cliques<<<G, 256, 0, s>>>(pe.roots.p, n, comp.p, ccount.p);
      k_root_flags<<<G, 256, 0, s>>>(comp.p, ccount.p, n, of_vertex, is_root.p, stats.p + 3 * ninst);
      count_launch(2);
    }
  }
  CDS_CUDA(cudaGetLastError());
  scan_u32(is_root.p, cidx.p, n, c, s);
  // The components' sizes, clique counts, largest core numbers and smallest vertices,
  // and local ids component by component (at most ncore of them).
  std::vector<uint64_t> hv;
  std::vector<unsigned long long> hc;
  uint32_t ncomp = 0;
  DBuf<uint32_t> csize(c, s, 0), cmax(c, s, 0), roots(c, s, 0), vcur(c, s, 0);
  DBuf<unsigned long long> cclq(c, s, 0);
  DBuf<uint64_t> vbeg(c, s, 0);
  auto tables = [&](uint32_t slots) {  // for up to that many components
    csize.alloc(slots);
    cmax.alloc(slots);
    roots.alloc(slots);
    vcur.alloc(slots);
    cclq.alloc(slots);
    vbeg.alloc(slots + 1);
    csize.zero();
    cclq.zero();
    cmax.zero();
    vcur.zero();
    k_comp_sizes<<<G, 256, 0, s>>>(comp.p, cidx.p, ccount.p, n, csize.p, cclq.p, pe.core.p, cmax.p);
    k_gather_roots<<<G, 256, 0, s>>>(is_root.p, cidx.p, n, roots.p);
    scan_u32(csize.p, vbeg.p, slots, c, s);
    out.vmap = DBuf<uint32_t>(c, s, ncore + 1);
    out.vcnet = DBuf<uint32_t>(c, s, ncore + 1);
    out.local = DBuf<uint32_t>(c, s, n + 1);
    k_local_ids<<<G, 256, 0, s>>>(comp.p, cidx.p, ccount.p, n, vbeg.p, vcur.p, out.local.p, out.vmap.p, out.vcnet.p);
    count_launch(3);
    CDS_CUDA(cudaGetLastError());
    hv.resize(slots + 1);
    hc.resize(slots);
    out.comp_maxcore.resize(slots);
    out.comp_root.resize(slots);
  };
  auto read_tables = [&](HostReads &r) {
    r.add(hv.data(), vbeg.p, hv.size());
    r.add(hc.data(), cclq.p, hc.size());
    r.add(out.comp_maxcore.data(), cmax.p, hc.size());
    r.add(out.comp_root.data(), roots.p, hc.size());
  };
  // One wait for the component count, the per-instance statistics and the status: of
  // a core of few vertices, which bound its components, also for the tables (24 bytes
  // a slot; a wait and the launches behind it cost about 15 us).
  const uint32_t early = ncore && ncore <= 1024 ? (uint32_t)ncore : 0u;
  if (early) tables(early);
  {
    uint64_t ncomp64 = 0;
    uint32_t e0 = 0;
    std::vector<unsigned long long> h(4 * (size_t)ninst);
    HostReads r(s);
    r.add(&ncomp64, cidx.p + n);
    r.add(&e0, err.p);
    r.add(h.data(), stats.p, h.size());
    if (early) read_tables(r);
    r.wait();
    out.core_size.assign(h.begin(), h.begin() + ninst);
    out.core_cliques.assign(h.begin() + ninst, h.begin() + 2 * ninst);
    out.pruned_edges.assign(h.begin() + 2 * ninst, h.begin() + 3 * ninst);
    out.n_components.resize(ninst);
    for (uint32_t i = 0; i < ninst; i++) out.n_components[i] = (uint32_t)h[3 * ninst + i];
    ncomp = (uint32_t)ncomp64;
    if (e0 & DEV_ERR_TIMEOUT) fail(CDS_ERR_TIMEOUT, "components: union-find retry budget exhausted");
    if (e0) fail(CDS_ERR_CUDA, "densest core: clique record is not a DAG path");
  }
  out.ncomp = ncomp;
  if (ncomp && !early) {
    tables(ncomp);
    HostReads r(s);
    read_tables(r);
    r.wait();
  }
  out.comp_inst.assign(ncomp, 0);
  out.comp_vbeg.assign(ncomp + 1, 0);
  out.comp_cbeg.assign(ncomp + 1, 0);
  out.comp_maxcore.resize(ncomp);
  out.comp_root.resize(ncomp);
  for (uint32_t i = 0; i < ncomp; i++) {
    out.comp_vbeg[i + 1] = (uint32_t)hv[i + 1];
    out.comp_cbeg[i + 1] = out.comp_cbeg[i] + hc[i];
    // instance of the root: binary search in the instance table
    out.comp_inst[i] = (uint32_t)(std::upper_bound(inst.h_vbeg.begin(), inst.h_vbeg.end(), out.comp_root[i]) -
                                  inst.h_vbeg.begin()) - 1;
  }
}

void build_networks(cds_ctx *c, cudaStream_t s, const Dag &gdag, uint32_t k, const Tuning &t, CoreOut &out,
                    const std::vector<uint8_t> &open, const CountHook *on_count) {
  const uint32_t ncomp = out.ncomp, nv = out.comp_vbeg[ncomp];
  const int G = c->sm_count * 8;
  if (!out.listed) {
    Dag dag;
    list_core_cliques(c, s, gdag, k, t, out, dag, on_count);
  }
  const uint64_t m = out.cliques.count;
  std::vector<uint64_t> hc(ncomp + 1, 0);  // first clique of each component's network
  for (uint32_t i = 0; i < ncomp; i++)
    hc[i + 1] = hc[i] + (open[i] ? out.comp_cbeg[i + 1] - out.comp_cbeg[i] : 0);
  const uint64_t nc = out.nc = hc[ncomp];
  DBuf<uint64_t> cbeg(c, s, ncomp + 1);
  DBuf<uint8_t> d_open(c, s, ncomp);
  CDS_CUDA(cudaMemcpyAsync(cbeg.p, hc.data(), (ncomp + 1) * 8, cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(d_open.p, open.data(), ncomp, cudaMemcpyHostToDevice, s));
  out.rec = DBuf<uint32_t>(c, s, (nc << rec_shift(k)) + 1);
  DBuf<uint32_t> ldeg(c, s, nv + 1);
  DBuf<unsigned long long> ccur(c, s, ncomp);
  ccur.zero();
  ldeg.zero();
  if (m) {
    ProfScope ps_b(c, s, "components_bucket");
    k_bucket_cliques<<<G, 256, 0, s>>>(out.cliques.members.p, m, k, out.comp.p, out.cidx.p, d_open.p, cbeg.p,
                                       ccur.p, out.local.p, nv, out.rec.p, ldeg.p);
    count_launch();
    CDS_CUDA(cudaGetLastError());
  }
  out.cliques.members.release();
  out.listed = false;
  out.vinc_off = DBuf<uint64_t>(c, s, nv + 1);
  scan_u32(ldeg.p, out.vinc_off.p, nv, c, s);
  out.flows_zero = true;
  // each vertex's cliques as u32 record indices while they fit, else u64
  // (two words each); the vertex's slot in a record is found by matching
  out.vinc_wide = nc >= 0xFFFFFFFFull || (c->flags & CDS_CONFIG_WIDE_FLOW);
  out.vinc = DBuf<uint32_t>(c, s, nc * k * (out.vinc_wide ? 2 : 1) + 2);
  {
    ProfScope ps_v(c, s, "components_vinc");
    DBuf<uint32_t> cur(c, s, nv + 1);
    cur.zero();
    if (nc && nv <= SMALL_NV && out.vinc_wide)
      k_fill_vinc_small<uint64_t><<<G, 256, 0, s>>>(out.rec.p, nc, k, nv, out.vinc_off.p, cur.p,
                                                    reinterpret_cast<uint64_t *>(out.vinc.p));
    else if (nc && nv <= SMALL_NV)
      k_fill_vinc_small<uint32_t><<<G, 256, 0, s>>>(out.rec.p, nc, k, nv, out.vinc_off.p, cur.p, out.vinc.p);
    else if (nc && out.vinc_wide)
      k_fill_vinc<uint64_t><<<G, 256, 0, s>>>(out.rec.p, nc, k, out.vinc_off.p, cur.p,
                                              reinterpret_cast<uint64_t *>(out.vinc.p));
    else if (nc)
      k_fill_vinc<uint32_t><<<G, 256, 0, s>>>(out.rec.p, nc, k, out.vinc_off.p, cur.p, out.vinc.p);
    count_launch();
    CDS_CUDA(cudaGetLastError());
  }
}

}  // namespace cds
