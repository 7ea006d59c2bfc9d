// peel.cu -- (k,Psi)-clique-core decomposition and the density of every core.
//
// Replaces cliqueCoreDecompose (cudaCode/main.cu:252-343) with selectNodes /
// processNodesByWarp (cudaCode/src/helpers.cu:611-750), whose removal step
// scans every clique for each removed vertex, and the serial oracle's peel
// (cpuCode/c++/src/helpers.cpp:16-150), which removes one minimum-degree
// vertex at a time and records the density of what is left.
//
// Core numbers as the fixpoint of a local operator instead of a peel.  For
// a vertex v with clique set Psi(v), let x_C = min over the other members u
// of C of tau(u).  H(v) = the largest h with at least h cliques x_C >= h.
// Starting from tau = clique degree (an upper bound of the core number),
// tau(v) <- H(v), applied in any order, decreases monotonically and stops
// exactly at the clique-core numbers: a fixpoint F satisfies F <= core (the
// vertices with F >= h span at least h cliques each inside that set, so they
// lie in the h-core), and every iterate stays >= core (H is monotone and
// core is its fixpoint).  This is the local characterisation of nucleus
// decompositions (Sariyuce, Seshadhri, Pinar, VLDB 2018) for 1-vertex
// nuclei of k-cliques.
//
// H without the cliques.  Order the vertices by tau (ties in any order) and give
// every clique to its first member, its root u.  Then x_C = tau(u) for every other member v of
// it, and x_C >= tau(u) for u itself, so
//     H(v) = the largest h <= tau(v) with R(v) + sum{ c(u,v) : tau(u) >= h } >= h
// where R(v) counts the cliques rooted at v and c(u,v) those rooted at u that
// hold v.  c(u,.) is what the counting pass computes from u's later neighbours
// N+(u) by bitmaps: 32 cliques an instruction, nothing stored per clique.  It
// depends on the set N+(u) alone, so a root is counted again only when a
// neighbour crossed it in the order.  With weights that are older than the
// values, tau(u) of the old root is at least the true x_C (it is one of the
// members the minimum is over), so an update with them is still an upper bound
// >= core: values may be lowered several times between two counts, and only a
// pass over current weights that lowers nothing ends the loop.
//
// Sweep (one cooperative launch, a grid barrier after each phase):
//   order   every vertex a change can have reached compares itself with its neighbours
//           before and after; where its later set changed, small sets are
//           counted at once by the warp, larger ones queued
//   count   blocks take the queued roots
//   lower   (LOWER times) weighted h-index of every vertex a change can have reached
// Ties keep the order they had: a vertex that arrives at a value goes behind those
// that were there (its key's low half holds the sweep it arrived in and how far
// it fell).  With ids to break ties a plateau of equal values turns around as it
// forms: R-MAT 200k k = 3 took 56 sweeps and 15 ms with ids, 46 and
// 10.4 ms this way.
// A change of a value from `old` to `new` reaches only vertices with new <= tau
// <= old: above old, both values are below tau; below new, the order around the
// vertex and the minimum with its own value stay as they were.
//
// Measured against sweeps over stored cliques (8-byte member tuples of every
// incidence, 17 to 21 passes): R-MAT scale 18, edge factor 16, k = 4 (2.29 G
// cliques, 9.1 G incidences) 605 ms for tuples and sweeps against 11 ms; R-MAT scale
// 16, edge factor 12, k = 4 37 against 2.1; R-MAT scale 14, edge factor 8: k = 4
// 2.2 against 1.0, k = 2 0.54 against 0.37.  Small graphs are bound by the chains
// of L2 reads in a phase and its barrier (about 50 us a sweep whatever the
// grid): k = 3 at scale 14 0.80 against 1.2.
//
// Densities: the alive set at each level of a peel is a core {v : core(v) >=
// L}; |V_L| and |Psi_L| come from two histograms by core number, of the vertices
// and of the cliques rooted at them (a root is a member of smallest core), and
// suffix sums; the best level keeps the first (smallest) L with the largest
// |Psi_L| / |V_L|, as the level-by-level peel records it.  Instances of a batch
// (disjoint vertex ranges) are independent and share every sweep.
#include "device_util.cuh"
#include "stages.h"

#include "list_kernels.cuh"

#include <algorithm>

namespace {

constexpr int THREADS = 512, WARPS = THREADS / 32;
// A row of more entries than this is a block's work, else a warp's.  Lowering takes
// the first (its searches walk a row several times); ordering the first where such
// rows are few (a block each, or two), else the second: a block's time on a row is a
// chain of L2 reads and synchronisations, and 16 warps take 16 rows meanwhile (R-MAT
// 200k k = 3: 2.9 -> 2.0 ms ordering, but 2.8 -> 3.2 ms lowering).
constexpr uint32_t ROW_FEW = 512, ROW_MANY = 2048;
constexpr uint32_t SEGMENT = 16384;   // row entries a block looks at before it writes positions
constexpr uint32_t WARP_SET = 32;     // later sets up to this size are counted by a warp at once
constexpr uint32_t BINS_WARP = 256, BINS_BLOCK = 1024;
// Lowering passes between two counts, while they lower anything.  A pass takes about 10 us,
// the counts of the generic K = 0 up to milliseconds a sweep (k = 6, random graph of 1,200
// vertices of degree 300: 2 passes 35.7 ms, 4 29.3, 8 25.4; R-MAT 8,192 k = 7 19.2, 16.0, 19.2).
template <int K>
constexpr int LOWER = K == 2 ? 1 : K == 0 ? 4 : 2;
constexpr uint32_t PAIR_ITEM = 64;    // later neighbours per item of a set too large for one team
constexpr int SLOTS = 4;              // control words of a phase, by its number modulo SLOTS

// control words: per lowering pass what changed, per sweep the queues
enum { P_LOW = 0, P_HIGH, P_WORDS = 32 };                  // P_LOW holds ~(smallest new value)
enum { Q_ROOTS = 0, Q_PAIRS, Q_NEXT_ROOT, Q_NEXT_PAIR, Q_WORDS = 32 };

struct CoreParams {
  uint32_t n, k;
  const uint64_t *off;      // [n+1] undirected rows
  const uint32_t *adj;      // [nnz]
  const uint32_t *rel;      // [nnz] position of the row's vertex in its neighbour's row
  ListParams dag;           // the degree-ordered DAG and heavy bitmap (counting)
  uint32_t *tau;            // [n] values now
  unsigned long long *key;  // [n] place in the order when it was last taken: value, then tie-break
  uint32_t *R;              // [n] cliques rooted at each vertex
  uint32_t *cin;            // [nnz] c(u, v) at the position of u in v's row
  uint32_t *later;          // [nnz] positions of a queued root's later neighbours, from its row start
  uint32_t *dplus;          // [n] how many
  const uint32_t *wide;     // [2 n] vertices with more than ROW_FEW (from n: ROW_MANY) neighbours
  const uint32_t *nwide;    // [2] how many
  uint32_t *queue;          // [n] roots to count
  uint2 *pairs;             // [..] (root, first of PAIR_ITEM later neighbours) of large sets
  uint32_t dmax;            // largest set a block counts by itself
  uint32_t *rows_global;    // rows outside shared memory (dmax > BLOCK_DMAX)
  uint64_t rows_slab;
  uint32_t *pass_ctl;       // [SLOTS * P_WORDS]
  uint32_t *sweep_ctl;      // [SLOTS * Q_WORDS]
  GridBarrier *bar;
  uint32_t *err;
  unsigned long long spin_limit;
  uint32_t max_sweeps;
  unsigned long long time_budget_ns;
  uint32_t *sweeps;         // sweeps run
  unsigned long long *phase_ns;  // [3] block 0's time per phase, barrier included (profiling; null: off)
};

// the order: keys, then ids
__device__ __forceinline__ bool after(unsigned long long kw, uint32_t w, unsigned long long ku, uint32_t u) {
  return kw > ku || (kw == ku && w > u);
}
// The key of a vertex of value t in this sweep's order, from its last one: the
// same while the value stands, else t, the sweep (up to 65,535) and on a log
// scale, 2,048 steps an octave, how far the value fell.
__device__ __forceinline__ unsigned long long key_now(unsigned long long key, uint32_t t, uint32_t sweep) {
  const uint32_t old = (uint32_t)(key >> 32);
  if (old == t) return key;
  uint32_t low = 0;
  if (sweep) {
    const uint32_t f = old - t, e = 31 - __clz(f | 1u);
    low = min(sweep, 65535u) << 16 | (e >= 11 ? e << 11 | ((f >> (e - 11)) & 2047u) : e << 11 | ((f << (11 - e)) & 2047u));
  }
  return (unsigned long long)t << 32 | low;
}
__device__ __forceinline__ unsigned long long key_of(const CoreParams &p, uint32_t v, uint32_t sweep) {
  return key_now(__ldcg(p.key + v), __ldcg(p.tau + v), sweep);
}

struct Range {  // of the changes since some point: [low new value, high old value]
  uint32_t lo, hi;
  __device__ __forceinline__ bool reaches(uint32_t t) const { return t >= lo && t <= hi; }
};
__device__ __forceinline__ Range pass_range(const uint32_t *pass_ctl, uint32_t pass) {
  const uint32_t *w = pass_ctl + (pass % SLOTS) * P_WORDS;
  return {~__ldcg(w + P_LOW), __ldcg(w + P_HIGH)};
}

// Calls visit(v, t) warp-uniformly for every vertex whose t = want(v), its value, is not 0,
// each by one warp.  A warp takes vertices a stride apart (ids correlate with degree in
// many graphs).  The first `busy` blocks have other work: they take none where the rest can
// hold the vertices 32 a warp.  (A phase of a small graph is a chain of L2 reads, so what a
// visit needs besides the row is asked for before it: a strip of 8,000 vertices, k = 3, 60.3
// -> 57.5 ms, a grid of 300 x 300 31.2 -> 28.9, R-MAT 16,384 0.78 -> 0.74.)
template <class Want, class Visit>
__device__ __forceinline__ void each_vertex(uint32_t n, uint32_t busy, Want want, Visit visit) {
  uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t skip = min(busy, gridDim.x / 2) * (blockDim.x >> 5);
  if (n <= 32 * (nwarps - skip)) {
    if (gwarp < skip) return;
    gwarp -= skip;
    nwarps -= skip;
  }
  const uint32_t per = min(32u, (n + nwarps - 1) / nwarps), groups = (n + per - 1) / per;
  for (uint32_t g = gwarp; g < groups; g += nwarps) {
    const uint64_t v64 = g + (uint64_t)lane_id() * groups;
    const uint32_t t = lane_id() < per && v64 < n ? want((uint32_t)v64) : 0u;
    for (uint32_t m = __ballot_sync(CDS_FULL, t != 0); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      visit(__shfl_sync(CDS_FULL, (uint32_t)v64, l), __shfl_sync(CDS_FULL, t, l));
    }
  }
}

// Order phase for entries i0 + lane, i0 + 32 + lane, ... (U of them) of u's row: which
// neighbours come after u now (bit x: the x-th), and whether any changed sides (in
// the first sweep, before which there is no order, all count as changed).  The
// counts of neighbours that went before u are cleared.
constexpr int ORDER_U = 8;
__device__ __forceinline__ uint32_t row_after(const CoreParams &p, uint32_t u, uint64_t b, uint32_t len,
                                              unsigned long long ku, unsigned long long nu, uint32_t sweep,
                                              uint32_t i0, bool &changed) {
  uint32_t w[ORDER_U], tw[ORDER_U], now = 0;
  unsigned long long kw[ORDER_U];
#pragma unroll
  for (int x = 0; x < ORDER_U; x++) w[x] = i0 + 32 * x < len ? __ldg(p.adj + b + i0 + 32 * x) : u;
#pragma unroll
  for (int x = 0; x < ORDER_U; x++) {
    tw[x] = __ldcg(p.tau + w[x]);
    kw[x] = __ldcg(p.key + w[x]);
  }
#pragma unroll
  for (int x = 0; x < ORDER_U; x++) {  // (past the end: u against itself, on neither side)
    const bool is = after(key_now(kw[x], tw[x], sweep), w[x], nu, u);
    const bool was = sweep ? after(kw[x], w[x], ku, u) : false;
    now |= is ? 1u << x : 0u;
    if (is != was) {
      changed = true;
      if (was) p.cin[p.off[w[x]] + __ldg(p.rel + b + i0 + 32 * x)] = 0;
    }
  }
  return now;
}

// The weights of root u over its counted later set (positions pos(r)).
template <int K, class Pos, class C>
__device__ __forceinline__ unsigned long long store_weights(const CoreParams &p, uint64_t b, uint32_t d, uint32_t tr,
                                                            uint32_t ts, Pos pos, const uint32_t *A, const C *cnt) {
  const uint32_t div = (K ? K : p.k) - 2;
  unsigned long long mine = 0;
  for (uint32_t r = tr; r < d; r += ts) {
    const uint32_t c = (uint32_t)(cnt[r] / div);
    mine += c;
    p.cin[p.off[A[r]] + __ldg(p.rel + b + pos(r))] = c;
  }
  return mine;
}

// Queues root u, whose later set (dplus, later) is in global memory.
__device__ __forceinline__ void queue_root(const CoreParams &p, uint32_t *sctl, uint32_t u, uint32_t d) {
  if (d <= p.dmax) {
    p.queue[atomicAdd(sctl + Q_ROOTS, 1u)] = u;
  } else {
    const uint32_t items = (d + PAIR_ITEM - 1) / PAIR_ITEM;
    const uint32_t at = atomicAdd(sctl + Q_PAIRS, items);
    for (uint32_t i = 0; i < items; i++) p.pairs[at + i] = make_uint2(u, i * PAIR_ITEM);
  }
}

// A set too small for a clique, or one whose items will add to its weights.
__device__ __forceinline__ void clear_weights(const CoreParams &p, uint32_t u, uint64_t b, uint32_t d, uint32_t tr,
                                              uint32_t ts) {
  for (uint32_t r = tr; r < d; r += ts) {
    const uint32_t i = __ldcg(p.later + b + r);
    p.cin[p.off[p.adj[b + i]] + p.rel[b + i]] = 0;
  }
  if (tr == 0) p.R[u] = 0;
}

// One item of a root whose later set is too large for a team: the cliques whose
// first member in the degree order is one of PAIR_ITEM later neighbours a, from
// the local graph of N+(a) inside the set (at most the DAG's largest out-degree).
template <int K>
__device__ void count_pairs(const CoreParams &p, uint2 item, uint32_t sweep, uint32_t *sm, uint32_t *rows) {
  using C = typename CountOf<K>::type;
  const uint32_t u = item.x, d = __ldcg(p.dplus + u);
  const unsigned long long nu = key_of(p, u, sweep);
  const uint64_t b = p.off[u];
  const uint32_t len = (uint32_t)(p.off[u + 1] - b), d4 = (p.dmax + 3) & ~3u;
  C *cnt = reinterpret_cast<C *>(sm);
  uint32_t *A = sm + d4 * (sizeof(C) / 4), *hid = A + d4;
  for (uint32_t r = item.y; r < min(d, item.y + PAIR_ITEM); r++) {
    const uint32_t ia = __ldcg(p.later + b + r), a = p.adj[b + ia];
    const uint32_t *list = p.dag.dadj + p.dag.doff[a];
    const uint32_t la = p.dag.outdeg[a];
    uint32_t m = 0;
    for (uint32_t i0 = 0; i0 < la; i0 += blockDim.x) {
      const uint32_t w = i0 + threadIdx.x < la ? list[i0 + threadIdx.x] : 0u;
      bool in = false;
      if (i0 + threadIdx.x < la && after(key_of(p, w, sweep), w, nu, u)) {
        uint32_t lo = 0, hi = len;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (p.adj[b + mid] < w) lo = mid + 1;
          else hi = mid;
        }
        in = lo < len && p.adj[b + lo] == w;
      }
      uint32_t total;
      const uint32_t at = m + block_exclusive_scan<uint32_t>(in ? 1u : 0u, &total);
      if (in) {
        A[at] = w;
        hid[at] = p.dag.heavy.id(w);
      }
      m += total;
    }
    __syncthreads();
    if (m == 0 || m < (K ? K : p.k) - 2) continue;
    unsigned long long mine = 0;
    if (K != 3) {
      constexpr int KS = K == 4 ? 3 : K == 5 ? 4 : 0;
      local_count<KS, true, C>(A, hid, m, p.dag.heavy, p.dag.doff, p.dag.dadj, p.dag.outdeg, rows, cnt,
                               (int)(K ? K : p.k) - 1);
    }
    const uint32_t div = K == 3 ? 1u : (K ? K : p.k) - 3;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
      const uint32_t c = K == 3 ? 1u : (uint32_t)(cnt[i] / div), w = A[i];
      mine += c;
      if (c) {
        uint32_t lo = 0, hi = len;  // w's position in u's row
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (p.adj[b + mid] < w) lo = mid + 1;
          else hi = mid;
        }
        atomicAdd(p.cin + p.off[w] + p.rel[b + lo], c);
      }
    }
    const unsigned long long total = Team<true>::sum<unsigned long long>(mine) / ((K ? K : p.k) - 2);
    if (threadIdx.x == 0 && total) {
      atomicAdd(p.cin + p.off[a] + p.rel[b + ia], (uint32_t)total);
      atomicAdd(p.R + u, (uint32_t)total);
    }
    __syncthreads();
  }
}

// Sum over a row of the weights whose value passes `test`, calling use(x, c) on
// the others; tr of ts threads take part, the sum is per thread.
template <int K, class Use>
__device__ __forceinline__ uint32_t row_sum(const CoreParams &p, uint64_t b, uint32_t len, uint32_t t, uint32_t tr,
                                            uint32_t ts, Use use) {
  constexpr int U = K == 2 ? 8 : 4;  // (k = 2 has no weights to keep: 8 entries, the star 8.5 -> 7.6 ms)
  uint32_t ge = 0;
  for (uint32_t i0 = tr; i0 < len; i0 += ts * U) {
    uint32_t w[U], c[U], x[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
      const bool in = i0 + ts * j < len;
      w[j] = in ? __ldg(p.adj + b + i0 + ts * j) : 0u;
      c[j] = !in ? 0u : K == 2 ? 1u : __ldcg(p.cin + b + i0 + ts * j);
    }
#pragma unroll
    for (int j = 0; j < U; j++) x[j] = c[j] ? __ldcg(p.tau + w[j]) : 0u;
#pragma unroll
    for (int j = 0; j < U; j++) {
      if (x[j] >= t) ge += c[j];
      else use(x[j], c[j]);
    }
  }
  return ge;
}

// Weighted h-index of a vertex whose weight S at values >= t falls short of t.
// S itself is feasible, so the answer lies in [lo, hi) = [S, t).  The weights in
// that range go into bins of 2^s values from hi - 1 down; the first bin whose
// lowest value has enough weight at or above it holds the answer, exactly for
// s = 0, and is the next range otherwise.  (A bound from one pass would do for
// the fixpoint, but many values just below t leave S far under the answer, and
// the sweeps then creep: 2,312 of them instead of 16 on R-MAT scale 18.)
struct BinSearch {
  uint32_t hi, lo, S, s;  // S: weight at values >= hi
  template <uint32_t BINS>
  __device__ __forceinline__ void shift() {
    s = 0;
    while (((hi - lo - 1) >> s) >= BINS) s++;
  }
  __device__ __forceinline__ bool holds(uint32_t x) const { return x >= lo && x < hi; }
  __device__ __forceinline__ uint32_t bin_of(uint32_t x) const { return (hi - 1 - x) >> s; }
  __device__ __forceinline__ void add(uint32_t *bin, uint32_t x, uint32_t c) const {
    if (holds(x) && c) atomicAdd(&bin[bin_of(x)], c);
  }
  // weight Sb at or above bin b's lowest value is enough (or that is below lo)
  __device__ __forceinline__ bool found(uint32_t b, uint32_t Sb) const {
    const unsigned long long down = (unsigned long long)(b + 1) << s;
    return down >= hi - lo || Sb >= (uint32_t)(hi - down);
  }
  // on to bin b, with the weight above it; true when hi - 1 is the answer
  __device__ __forceinline__ bool narrow(uint32_t b, uint32_t above_b) {
    const unsigned long long down = (unsigned long long)(b + 1) << s;
    if (down < hi - lo) lo = hi - (uint32_t)down;
    hi -= b << s;
    S = above_b;
    return s == 0;
  }
};

template <int K>
__device__ __forceinline__ uint32_t lower_warp(const CoreParams &p, uint32_t v, uint32_t t, uint32_t *bin) {
  const uint32_t lane = lane_id();
  const uint64_t b = p.off[v];
  const uint32_t len = (uint32_t)(p.off[v + 1] - b), rooted = K == 2 ? 0u : __ldcg(p.R + v);
  uint32_t ge = row_sum<K>(p, b, len, t, lane, 32, [](uint32_t, uint32_t) {});
  ge = __reduce_add_sync(CDS_FULL, ge) + rooted;
  if (ge >= t) return t;
  BinSearch bs{t, ge, ge, 0};
  for (;;) {
    bs.shift<BINS_WARP>();
    for (uint32_t i = lane; i < BINS_WARP; i += 32) bin[i] = 0;
    __syncwarp();
    row_sum<K>(p, b, len, 0xFFFFFFFFu, lane, 32, [&](uint32_t x, uint32_t c) { bs.add(bin, x, c); });
    __syncwarp();
    uint32_t base = bs.S, m = 0, S = 0, x = 0, b0 = 0;
    for (;; b0 += 32) {  // the last bin reaches lo, so some bin is found
      x = bin[b0 + lane];
      S = base + warp_inclusive_scan(x);
      m = __ballot_sync(CDS_FULL, bs.found(b0 + lane, S));
      if (m) break;
      base = __shfl_sync(CDS_FULL, S, 31);
    }
    const uint32_t at = __ffs(m) - 1;
    const bool exact = bs.narrow(b0 + at, __shfl_sync(CDS_FULL, S - x, at));
    __syncwarp();  // the bins are reused
    if (exact) return bs.hi - 1;
  }
}

template <int K>
__device__ __forceinline__ uint32_t lower_block(const CoreParams &p, uint32_t v, uint32_t t, uint32_t *bin) {
  __shared__ uint32_t s_first, s_above;
  const uint64_t b = p.off[v];
  const uint32_t len = (uint32_t)(p.off[v + 1] - b);
  const uint32_t mine = row_sum<K>(p, b, len, t, threadIdx.x, blockDim.x, [](uint32_t, uint32_t) {});
  uint32_t ge;
  block_exclusive_scan<uint32_t>(mine, &ge);
  ge += K == 2 ? 0u : __ldcg(p.R + v);
  if (ge >= t) return t;
  BinSearch bs{t, ge, ge, 0};
  for (;;) {
    bs.shift<BINS_BLOCK>();
    for (uint32_t i = threadIdx.x; i < BINS_BLOCK; i += blockDim.x) bin[i] = 0;
    if (threadIdx.x == 0) s_first = 0xFFFFFFFFu;
    __syncthreads();
    // (a hub's neighbours are mostly of a few small values, so a thread adds up a bin's
    // weights while they come: a star of 4 M vertices, k = 2, 12.1 -> 8.5 ms)
    uint32_t at = 0, sum = 0;
    row_sum<K>(p, b, len, 0xFFFFFFFFu, threadIdx.x, blockDim.x, [&](uint32_t x, uint32_t c) {
      if (!bs.holds(x) || !c) return;
      if (bs.bin_of(x) != at) {
        if (sum) atomicAdd(&bin[at], sum);
        at = bs.bin_of(x);
        sum = 0;
      }
      sum += c;
    });
    if (sum) atomicAdd(&bin[at], sum);
    __syncthreads();
    static_assert(BINS_BLOCK == 2 * THREADS, "two bins a thread");
    const uint32_t b0 = 2 * threadIdx.x, x0 = bin[b0], x1 = bin[b0 + 1];
    uint32_t total;
    const uint32_t S0 = bs.S + block_exclusive_scan<uint32_t>(x0 + x1, &total) + x0, S1 = S0 + x1;
    const bool f0 = bs.found(b0, S0), f1 = bs.found(b0 + 1, S1);
    if (f0 || f1) atomicMin(&s_first, f0 ? b0 : b0 + 1);
    __syncthreads();
    if (s_first / 2 == threadIdx.x) s_above = s_first == b0 ? S0 - x0 : S0;
    __syncthreads();
    const bool exact = bs.narrow(s_first, s_above);
    __syncthreads();  // s_first, s_above and the bins are reused
    if (exact) return bs.hi - 1;
  }
}

// shared words a warp uses in the order phase: counts, set, heavy ids, rows of up to
// WARP_SET vertices, and the sides of a row
template <class C>
constexpr uint32_t ORDER_WORDS = (sizeof(C) / 4 + 3) * WARP_SET + ROW_MANY / 32;

template <int K>
__global__ void __launch_bounds__(THREADS, 2) k_core(CoreParams p) {
  using C = typename CountOf<K>::type;
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint32_t s_low, s_high, s_item;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  const unsigned long long t0 = globaltimer_ns();
  const uint32_t nlong = p.nwide[0];
  const bool many = nlong > 2 * gridDim.x;
  const uint32_t nwide = p.nwide[many ? 1 : 0], row_max = many ? ROW_MANY : ROW_FEW;
  const uint32_t *wide = p.wide + (many ? p.n : 0), kmin = (K ? K : p.k) - 1;
  if (threadIdx.x == 0) {
    s_low = 0;
    s_high = 0;
  }
  __syncthreads();
  uint32_t pass = 0, sweep = 0;
  bool done = false;
  Range moved{0u, 0xFFFFFFFFu};
  unsigned long long tprev = t0;
  auto phase_end = [&](int i) {
    if (p.phase_ns && leader) {
      const unsigned long long now = globaltimer_ns();
      p.phase_ns[i] += now - tprev;
      tprev = now;
    }
  };
  for (; sweep < p.max_sweeps && !done; sweep++) {
    if (leader && globaltimer_ns() - t0 > p.time_budget_ns) atomicOr(p.err, DEV_ERR_TIMEOUT);
    // what changed since the vertices were last ordered (all of it, at first)
    const Range since = moved;
    moved = Range{0xFFFFFFFFu, 0u};
    if constexpr (K != 2) {
      uint32_t *sctl = p.sweep_ctl + (sweep % SLOTS) * Q_WORDS;
      if (leader)  // of the next sweep: no block reads or writes them in this one
        for (int i = 0; i < 4; i++) p.sweep_ctl[((sweep + 1) % SLOTS) * Q_WORDS + i] = 0;
      // ---- order: long rows by blocks, then the others by warps.  One look at a
      // row gives the side of every entry, as words in shared memory; positions
      // are written from them.
      for (uint32_t x = blockIdx.x; x < nwide; x += gridDim.x) {
        const uint32_t u = wide[x], t = __ldcg(p.tau + u);
        if (t == 0 || !since.reaches(t)) continue;
        const uint64_t b = p.off[u];
        const uint32_t len = (uint32_t)(p.off[u + 1] - b);
        const unsigned long long ku = __ldcg(p.key + u), nu = key_now(ku, t, sweep);
        uint32_t d = 0;
        bool changed = false;
        for (uint32_t s0 = 0; s0 < len; s0 += SEGMENT) {
          const uint32_t n = min(SEGMENT, len - s0);
          for (uint32_t i0 = warp * 32 * ORDER_U; i0 < n; i0 += THREADS * ORDER_U) {
            const uint32_t now = row_after(p, u, b, s0 + n, ku, nu, sweep, s0 + i0 + lane, changed);
#pragma unroll
            for (int y = 0; y < ORDER_U; y++) {
              const uint32_t m = __ballot_sync(CDS_FULL, (now >> y) & 1u);
              if (lane == y) sm[(i0 >> 5) + y] = m;  // (SEGMENT is a multiple of the step)
            }
          }
          __syncthreads();
          uint32_t m = threadIdx.x < (n + 31) / 32 ? sm[threadIdx.x] : 0u, total;
          static_assert(SEGMENT / 32 == THREADS, "a word a thread");
          uint32_t at = d + block_exclusive_scan<uint32_t>(__popc(m), &total);
          for (; m; m &= m - 1) p.later[b + at++] = s0 + threadIdx.x * 32 + __ffs(m) - 1;
          d += total;
        }
        if (!__syncthreads_or(changed)) continue;  // (and the list, for the block's own reads below)
        if (threadIdx.x == 0) p.dplus[u] = d;
        if (d < kmin || d > p.dmax) clear_weights(p, u, b, d, threadIdx.x, blockDim.x);
        if (d >= kmin && threadIdx.x == 0) queue_root(p, sctl, u, d);
      }
      __syncthreads();
      {
        constexpr uint32_t CW = sizeof(C) / 4, MW = ROW_MANY / 32;
        uint32_t *area = sm + warp * ORDER_WORDS<C>;
        C *cnt = reinterpret_cast<C *>(area);
        uint32_t *A = area + CW * WARP_SET, *hid = A + WARP_SET, *rows = hid + WARP_SET, *side = rows + WARP_SET;
        each_vertex(
            p.n, nwide,
            [&](uint32_t v) {
              const uint32_t t = __ldcg(p.tau + v);
              return t && since.reaches(t) && p.off[v + 1] - p.off[v] <= row_max ? t : 0u;
            },
            [&](uint32_t u, uint32_t t) {
              const uint64_t b = p.off[u];
              const uint32_t len = (uint32_t)(p.off[u + 1] - b);
              const unsigned long long ku = __ldcg(p.key + u), nu = key_now(ku, t, sweep);
              bool changed = false;
              for (uint32_t i0 = 0; i0 < len; i0 += 32 * ORDER_U) {
                const uint32_t now = row_after(p, u, b, len, ku, nu, sweep, i0 + lane, changed);
#pragma unroll
                for (int y = 0; y < ORDER_U; y++) {
                  const uint32_t m = __ballot_sync(CDS_FULL, (now >> y) & 1u);
                  if (lane == y) side[(i0 >> 5) + y] = m;
                }
              }
              if (!__any_sync(CDS_FULL, changed)) return;
              __syncwarp();
              // lane l holds words l and l + 32 of the row's sides
              static_assert(MW == 64, "two words a lane");
              const uint32_t nw = (len + 31) / 32;
              const uint32_t m0 = lane < nw ? side[lane] : 0u, m1 = lane + 32 < nw ? side[lane + 32] : 0u;
              const uint32_t i0 = warp_inclusive_scan((uint32_t)__popc(m0)), n0 = __shfl_sync(CDS_FULL, i0, 31);
              const uint32_t i1 = n0 + warp_inclusive_scan((uint32_t)__popc(m1)), d = __shfl_sync(CDS_FULL, i1, 31);
              uint32_t at = i0 - __popc(m0);
              for (uint32_t m = m0; m; m &= m - 1) p.later[b + at++] = lane * 32 + __ffs(m) - 1;
              at = i1 - __popc(m1);
              for (uint32_t m = m1; m; m &= m - 1) p.later[b + at++] = (lane + 32) * 32 + __ffs(m) - 1;
              __syncwarp();
              if (d < kmin) {
                clear_weights(p, u, b, d, lane, 32);
              } else if (d <= WARP_SET) {
                const uint32_t pos = lane < d ? __ldcg(p.later + b + lane) : 0u;
                if (lane < d) {
                  const uint32_t a = p.adj[b + pos];
                  A[lane] = a;
                  hid[lane] = p.dag.heavy.id(a);
                }
                __syncwarp();
                local_count<K, false, C, true>(A, hid, d, p.dag.heavy, p.dag.doff, p.dag.dadj, p.dag.outdeg,
                                               rows, cnt, (int)kmin + 1);
                const unsigned long long total =
                    warp_sum(store_weights<K>(p, b, d, lane, 32, [&](uint32_t) { return pos; }, A, cnt)) / kmin;
                if (lane == 0) p.R[u] = (uint32_t)total;
                __syncwarp();
              } else {
                if (d > p.dmax) clear_weights(p, u, b, d, lane, 32);  // (its items add to them)
                if (lane == 0) {
                  p.dplus[u] = d;
                  queue_root(p, sctl, u, d);
                }
              }
            });
      }
      if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
      phase_end(0);
      // ---- count: the queued roots by blocks
      {
        const uint32_t nroots = __ldcg(sctl + Q_ROOTS), npairs = __ldcg(sctl + Q_PAIRS);
        const uint32_t d4 = (p.dmax + 3) & ~3u;
        C *cnt = reinterpret_cast<C *>(sm);
        uint32_t *A = sm + d4 * (sizeof(C) / 4), *hid = A + d4;
        uint32_t *rows = p.rows_global ? p.rows_global + (uint64_t)blockIdx.x * p.rows_slab : hid + d4;
        for (int kind = 0; kind < 2; kind++) {
          const uint32_t total_items = kind ? npairs : nroots;
          for (uint32_t r = blockIdx.x; r < total_items;) {
            if (kind) {
              count_pairs<K>(p, __ldcg(p.pairs + r), sweep, sm, rows);
            } else {
              const uint32_t u = __ldcg(p.queue + r), d = __ldcg(p.dplus + u);
              const uint64_t b = p.off[u];
              for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) {
                const uint32_t a = p.adj[b + __ldcg(p.later + b + i)];
                A[i] = a;
                hid[i] = p.dag.heavy.id(a);
              }
              __syncthreads();
              local_count<K, true, C>(A, hid, d, p.dag.heavy, p.dag.doff, p.dag.dadj, p.dag.outdeg,
                                                   rows, cnt, (int)kmin + 1);
              const unsigned long long total =
                  Team<true>::sum<unsigned long long>(store_weights<K>(
                      p, b, d, threadIdx.x, blockDim.x,
                      [&](uint32_t i) { return __ldcg(p.later + b + i); }, A, cnt)) / kmin;
              if (threadIdx.x == 0) p.R[u] = (uint32_t)total;
            }
            // the first items go by block number, the rest by a counter
            if (threadIdx.x == 0) s_item = gridDim.x + atomicAdd(sctl + (kind ? Q_NEXT_PAIR : Q_NEXT_ROOT), 1u);
            __syncthreads();
            r = s_item;
            __syncthreads();
          }
        }
      }
      // (every block read the same sizes; with nothing queued nothing was written)
      if (__ldcg(sctl + Q_ROOTS) + __ldcg(sctl + Q_PAIRS) && !grid_sync(p.bar, p.err, p.spin_limit)) return;
      phase_end(1);
    }
    // ---- lower
    Range reach = since;
    for (int x = 0; x < LOWER<K>; x++) {
      uint32_t *pctl = p.pass_ctl + (pass % SLOTS) * P_WORDS;
      if (leader)  // of the next pass: last read two passes ago
        for (int i = 0; i < 2; i++) p.pass_ctl[((pass + 1) % SLOTS) * P_WORDS + i] = 0;
      for (uint32_t i = blockIdx.x; i < nlong; i += gridDim.x) {
        const uint32_t v = p.wide[i], t = __ldcg(p.tau + v);
        if (t == 0 || !reach.reaches(t)) continue;
        const uint32_t nt = lower_block<K>(p, v, t, sm);
        if (threadIdx.x == 0) {
          if (x == 0 && K != 2) p.key[v] = key_now(__ldcg(p.key + v), t, sweep);
          if (nt < t) {
            p.tau[v] = nt;
            atomicMax(&s_low, ~nt);
            atomicMax(&s_high, t);
          }
        }
      }
      __syncthreads();
      each_vertex(
          p.n, nlong,
          [&](uint32_t v) {
            const uint32_t t = __ldcg(p.tau + v);
            return t && reach.reaches(t) && p.off[v + 1] - p.off[v] <= ROW_FEW ? t : 0u;
          },
          [&](uint32_t v, uint32_t t) {
            const unsigned long long kv = x == 0 && K != 2 ? __ldcg(p.key + v) : 0ull;
            const uint32_t nt = lower_warp<K>(p, v, t, sm + warp * BINS_WARP);
            if (lane == 0) {
              if (x == 0 && K != 2) p.key[v] = key_now(kv, t, sweep);
              if (nt < t) {
                p.tau[v] = nt;
                atomicMax(&s_low, ~nt);
                atomicMax(&s_high, t);
              }
            }
          });
      __syncthreads();
      if (threadIdx.x == 0 && s_high) {
        atomicMax(pctl + P_LOW, s_low);
        atomicMax(pctl + P_HIGH, s_high);
        s_low = 0;
        s_high = 0;
      }
      if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
      phase_end(2);
      reach = pass_range(p.pass_ctl, pass++);
      moved.lo = min(moved.lo, reach.lo);
      moved.hi = max(moved.hi, reach.hi);
      if (reach.lo > reach.hi) {  // nothing lowered: with current weights (x = 0) that is the end
        done = x == 0;
        break;
      }
    }
  }
  if (leader) {
    *p.sweeps = sweep;
    if (!done) atomicOr(p.err, DEV_ERR_TIMEOUT);
  }
}

// rel[e], for e = the position of w in u's row: the position of u in w's row.
// Each edge once, from its end of larger (degree, id), searching the shorter row.
__global__ void k_rel(const uint64_t *__restrict__ off, const uint32_t *__restrict__ adj, uint32_t n, uint64_t nnz,
                      uint32_t *__restrict__ rel) {
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * 32 < nnz; c += warps) {
    uint32_t lo = 0, hi = n;  // the row of the first of 32 arcs
    while (hi - lo > 1) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (off[mid] <= c * 32) lo = mid;
      else hi = mid;
    }
    const uint64_t e = c * 32 + lane_id();
    if (e >= nnz) continue;
    // this arc's row: mostly that one or one of the next, but a run of empty rows between
    // may be as long as the graph (20 M of them, walked one by one: 1.8 s)
    uint32_t u = lo, last = lo;  // off[u] <= e; last + 1: the first row tried that ends past e
    for (uint32_t step = 1; off[last + 1] <= e; step *= 2) {
      u = last + 1;
      last = n - 1 - last > step ? last + step : n - 1;
    }
    while (u < last) {
      const uint32_t mid = u + (last - u) / 2;
      if (off[mid + 1] <= e) u = mid + 1;
      else last = mid;
    }
    const uint32_t w = adj[e];
    const uint64_t bu = off[u], bw = off[w];
    const uint32_t du = (uint32_t)(off[u + 1] - bu), dw = (uint32_t)(off[w + 1] - bw);
    if (!above(du, u, dw, w)) continue;
    uint32_t a = 0, z = dw;
    while (a < z) {
      const uint32_t mid = (a + z) >> 1;
      if (adj[bw + mid] < u) a = mid + 1;
      else z = mid;
    }
    rel[e] = a;
    rel[bw + a] = (uint32_t)(e - bu);
  }
}

__global__ void k_wide(const uint64_t *__restrict__ off, uint32_t n, uint32_t *__restrict__ wide,
                       uint32_t *__restrict__ nwide) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint64_t d = off[v + 1] - off[v];
    if (d > ROW_FEW) wide[atomicAdd(nwide, 1u)] = v;
    if (d > ROW_MANY) wide[n + atomicAdd(nwide + 1, 1u)] = v;
  }
}

// largest core per instance and the vertex histogram of core numbers
__global__ void k_inst_maxcore(const uint32_t *__restrict__ core, uint32_t n,
                               const uint32_t *__restrict__ of_vertex, uint32_t *__restrict__ out) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t v = base + threadIdx.x;
    const bool ok = v < n;
    const uint32_t key = ok ? (of_vertex ? of_vertex[v] : 0u) : 0xFFFFFFFFu;
    const uint32_t grp = __match_any_sync(CDS_FULL, key);
    const uint32_t m = __reduce_max_sync(grp, ok ? core[v] : 0u);
    if (ok && (__ffs(grp) - 1) == (int)lane_id()) atomicMax(out + key, m);
  }
}

// hv[hoff[i] + L] = vertices of instance i with core L, hc likewise the cliques
// rooted at them (k = 2: a vertex roots the edges to later neighbours)
__global__ void k_core_hist(const uint32_t *__restrict__ core, const uint32_t *__restrict__ R, uint32_t n,
                            const uint32_t *__restrict__ of_vertex, const uint64_t *__restrict__ hoff,
                            unsigned long long *__restrict__ hv, unsigned long long *__restrict__ hc,
                            uint32_t *__restrict__ used) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t v = base + threadIdx.x;
    const bool ok = v < n;
    uint64_t key = ~0ull;
    if (ok) key = hoff[of_vertex ? of_vertex[v] : 0u] + core[v];
    const uint32_t grp = __match_any_sync(CDS_FULL, key);
    if (ok && (__ffs(grp) - 1) == (int)lane_id()) {
      atomicAdd(hv + key, (unsigned long long)__popc(grp));
      if (used) used[key] = 1;
    }
    if (ok && R[v]) atomicAdd(hc + key, (unsigned long long)R[v]);
  }
}
__global__ void k_edge_roots(const uint64_t *__restrict__ off, const uint32_t *__restrict__ adj,
                             const uint32_t *__restrict__ core, uint32_t n, uint32_t *__restrict__ R) {
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
    const uint32_t t = core[v];
    uint32_t c = 0;
    for (uint64_t i = off[v] + lane_id(); i < off[v + 1]; i += 32) {
      const uint32_t w = adj[i], tw = core[w];
      c += tw > t || (tw == t && w > v);
    }
    c = __reduce_add_sync(CDS_FULL, c);
    if (lane_id() == 0) R[v] = c;
  }
}

// Long histograms are mostly empty: the bins in use, in order, and their values of L
// (pos: the bins in use before each).  One block takes 3.6 us for 4,096 bins, the scan
// and this about 25 us: worth it from LEVELS_DIRECT bins on (2.2 M bins, 11,125 in
// use: 1.96 -> 0.09 ms).
constexpr uint64_t LEVELS_DIRECT = 32768;
__global__ void k_levels_in_use(const uint32_t *__restrict__ used, const uint64_t *__restrict__ pos, uint64_t bins,
                                const uint64_t *__restrict__ hoff, uint32_t ninst,
                                const unsigned long long *__restrict__ hv, const unsigned long long *__restrict__ hc,
                                uint64_t *__restrict__ off, unsigned long long *__restrict__ v,
                                unsigned long long *__restrict__ cl, uint32_t *__restrict__ lvl) {
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = t0; i <= ninst; i += stride) off[i] = pos[hoff[i]];
  for (uint64_t b = t0; b < bins; b += stride) {
    if (!used[b]) continue;
    uint32_t lo = 0, hi = ninst;  // its instance: the last with hoff <= b
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (hoff[mid] <= b) lo = mid;
      else hi = mid;
    }
    v[pos[b]] = hv[b];
    cl[pos[b]] = hc[b];
    lvl[pos[b]] = (uint32_t)(b - hoff[lo]);
  }
}

// One block per instance: suffix sums over L of both histograms give the
// core {core >= L}; keep the smallest L of largest density (the first level
// a peel would record), and count the distinct core numbers.
__global__ void __launch_bounds__(512) k_best_level(const uint64_t *__restrict__ hoff,
                                                    const unsigned long long *__restrict__ hv,
                                                    const unsigned long long *__restrict__ hc,
                                                    const uint32_t *__restrict__ lvl,  // bins' L (null: all bins)
                                                    uint32_t ninst, unsigned long long *__restrict__ best_num,
                                                    unsigned long long *__restrict__ best_den,
                                                    uint32_t *__restrict__ levels,
                                                    uint32_t *__restrict__ best_lvl) {
  __shared__ unsigned long long s_v, s_c;
  __shared__ unsigned long long s_bn[16], s_bd[16];
  __shared__ uint32_t s_lv[16], s_bl[16];
  for (uint32_t i = blockIdx.x; i < ninst; i += gridDim.x) {
    const uint64_t b = hoff[i], nb = hoff[i + 1] - b;
    if (threadIdx.x == 0) {
      s_v = 0;
      s_c = 0;
    }
    __syncthreads();
    unsigned long long bn = 0, bd = 0;
    uint32_t lv = 0, bl = 0;  // bl: the level of (bn, bd)
    // chunks of blockDim * LEVEL_ITEMS bins from the top (largest L) down;
    // thread t holds LEVEL_ITEMS consecutive bins below those of thread t-1
    constexpr int LEVEL_ITEMS = 8;
    for (uint64_t top = nb; top > 0;) {
      const uint64_t span = (uint64_t)blockDim.x * LEVEL_ITEMS;
      const uint64_t lo = top > span ? top - span : 0;
      const uint64_t first = top - 1 - (uint64_t)threadIdx.x * LEVEL_ITEMS;  // this thread's top bin
      unsigned long long xv[LEVEL_ITEMS], xc[LEVEL_ITEMS], tv = 0, tc = 0;
#pragma unroll
      for (int j = 0; j < LEVEL_ITEMS; j++) {
        const uint64_t L = first - j;
        const bool in = (uint64_t)threadIdx.x * LEVEL_ITEMS + j < top - lo;  // L in [lo, top)
        xv[j] = in ? hv[b + L] : 0;
        xc[j] = in ? hc[b + L] : 0;
        tv += xv[j];
        tc += xc[j];
      }
      unsigned long long chunk_v, chunk_c;
      // suffix sums above this thread's first bin
      unsigned long long sv = block_exclusive_scan<unsigned long long>(tv, &chunk_v) + s_v;
      unsigned long long sc = block_exclusive_scan<unsigned long long>(tc, &chunk_c) + s_c;
#pragma unroll
      for (int j = 0; j < LEVEL_ITEMS; j++) {
        sv += xv[j];
        sc += xc[j];
        if (xv[j]) {  // a level with vertices (bins outside [lo, top) hold 0)
          lv++;
          // sc/sv > bn/bd, or equal with a smaller L (later in this loop)
          const unsigned long long lh = __umul64hi(sc, bd), ll = sc * bd;
          const unsigned long long rh = __umul64hi(bn, sv), rl = bn * sv;
          if (bd == 0 || lh > rh || (lh == rh && ll >= rl)) {
            bn = sc;
            bd = sv;
            bl = (uint32_t)(first - j);
          }
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        s_v += chunk_v;
        s_c += chunk_c;
      }
      __syncthreads();
      top = lo;
    }
    // the block's best: largest density, then smallest L; every thread's
    // candidate has the smallest L among its ties, and L falls with the
    // thread's progress, so among equal densities the larger sv wins
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long on = __shfl_down_sync(CDS_FULL, bn, o);
      const unsigned long long od = __shfl_down_sync(CDS_FULL, bd, o);
      const uint32_t ol = __shfl_down_sync(CDS_FULL, bl, o);
      lv += __shfl_down_sync(CDS_FULL, lv, o);
      if (od) {
        const unsigned long long lh = __umul64hi(on, bd), ll = on * bd;
        const unsigned long long rh = __umul64hi(bn, od), rl = bn * od;
        const bool gt = lh > rh || (lh == rh && ll > rl);
        const bool eq = lh == rh && ll == rl;
        if (bd == 0 || gt || (eq && od > bd)) {
          bn = on;
          bd = od;
          bl = ol;
        }
      }
    }
    if (lane_id() == 0) {
      s_bn[threadIdx.x >> 5] = bn;
      s_bd[threadIdx.x >> 5] = bd;
      s_lv[threadIdx.x >> 5] = lv;
      s_bl[threadIdx.x >> 5] = bl;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long fn = 0, fd = 0;
      uint32_t fl = 0, fb = 0;
      for (uint32_t w = 0; w < (blockDim.x >> 5); w++) {
        fl += s_lv[w];
        const unsigned long long on = s_bn[w], od = s_bd[w];
        if (!od) continue;
        const unsigned long long lh = __umul64hi(on, fd), ll = on * fd;
        const unsigned long long rh = __umul64hi(fn, od), rl = fn * od;
        const bool gt = lh > rh || (lh == rh && ll > rl);
        const bool eq = lh == rh && ll == rl;
        if (fd == 0 || gt || (eq && od > fd)) {
          fn = on;
          fd = od;
          fb = s_bl[w];
        }
      }
      best_num[i] = fn;
      best_den[i] = fd;
      levels[i] = fl;
      best_lvl[i] = fd && lvl ? lvl[b + fb] : fb;
    }
    __syncthreads();
  }
}

}  // namespace

namespace cds {

void peel(cds_ctx *c, cudaStream_t s, const uint64_t *off, const uint32_t *adj, uint64_t nnz, const Dag &dag,
          const Cliques &cl, const Instances &inst, uint32_t gl_buffer_size, PeelOut &out) {
  const uint32_t n = dag.n, k = cl.k;
  const uint64_t m = cl.count;
  const uint32_t ninst = inst.count;
  const uint32_t *of_vertex = ninst > 1 ? inst.of_vertex.p : nullptr;
  (void)gl_buffer_size;  // the reference's per-block removal buffer length has no counterpart
  out.core.c = c;
  out.core.s = s;
  out.core.alloc(n + 1);
  out.best_num.assign(ninst, 0);
  out.best_den.assign(ninst, 0);
  out.inst_max_core.assign(ninst, 0);
  out.inst_levels.assign(ninst, 0);
  out.best_level.assign(ninst, 0);
  out.levels = 0;
  out.max_core = 0;
  if (n == 0) return;
  DBuf<unsigned long long> phase(c, s, c->prof ? 3 : 0);
  phase.zero();
  CDS_CUDA(cudaMemcpyAsync(out.core.p, cl.cdeg.p, (size_t)n * 4, cudaMemcpyDeviceToDevice, s));

  // work words in one zeroed block: barrier, status, control slots, queue sizes
  constexpr size_t CTL = 32 + SLOTS * (P_WORDS + Q_WORDS) + 4;  // nwide[2], sweeps, err
  DBuf<uint32_t> ctl(c, s, CTL), wide(c, s, 2 * (size_t)n);
  out.roots.c = c;
  out.roots.s = s;
  out.roots.alloc(n + 1);
  DBuf<uint32_t> &R = out.roots;
  ctl.zero();
  R.zero();
  uint32_t *const ctl_err = ctl.p + CTL - 1, *const ctl_sweeps = ctl.p + CTL - 2, *const ctl_nwide = ctl.p + CTL - 4;
  k_wide<<<c->sm_count * 2, 256, 0, s>>>(off, n, wide.p, ctl_nwide);
  count_launch();
  {
    CoreParams p{};
    p.n = n;
    p.k = k;
    p.off = off;
    p.adj = adj;
    p.tau = out.core.p;
    p.R = R.p;
    p.wide = wide.p;
    p.nwide = ctl_nwide;
    static_assert(sizeof(GridBarrier) == 32 * sizeof(uint32_t), "the barrier takes the first line");
    p.bar = reinterpret_cast<GridBarrier *>(ctl.p);
    p.pass_ctl = ctl.p + 32;
    p.sweep_ctl = p.pass_ctl + SLOTS * P_WORDS;
    p.err = ctl_err;
    p.sweeps = ctl_sweeps;
    p.phase_ns = phase.p;
    p.spin_limit = 1ull << 26;
    p.max_sweeps = 1u << 20;
    p.time_budget_ns = 120ull * 1000000000ull;
    DBuf<unsigned long long> key(c, s, 0);
    DBuf<uint32_t> rel(c, s, 0), cin(c, s, 0), later(c, s, 0), dplus(c, s, 0), queue(c, s, 0),
        rows(c, s, 0);
    DBuf<uint2> pairs(c, s, 0);
    size_t smem = (size_t)std::max<uint32_t>(WARPS * BINS_WARP, BINS_BLOCK) * 4;
    unsigned blocks = coop_grid(c, 2);
    if (k >= 3 && m) {
      rel.alloc(nnz + 1);
      key.alloc(n);
      cin.alloc(nnz + 1);
      later.alloc(nnz + 1);
      dplus.alloc(n);
      queue.alloc(n);
      cin.zero();
      key.zero();  // (read for vertices in no clique, which are never ordered)
      {
        ProfScope ps(c, s, "peel_arcs");
        k_rel<<<c->sm_count * 8, 256, 0, s>>>(off, adj, n, nnz, rel.p);
        count_launch();
        CDS_CUDA(cudaGetLastError());
      }
      // the largest later set one block counts: as far as two blocks' rows fit
      // an SM (768: 95 KB), or the DAG's largest out-degree where that is more
      // (count_pairs needs it); past BLOCK_DMAX the rows go to global memory
      const int K = k <= 5 ? (int)k : 0;
      p.dmax = std::max<uint32_t>(k == 3 ? 4096 : 768, dag.max_out);
      const bool rows_in_smem = k == 3 || p.dmax <= (uint32_t)BLOCK_DMAX;
      if (!rows_in_smem) {
        p.rows_slab = rows_slab_words(p.dmax);
        blocks = std::min<unsigned>(blocks, coop_grid(c, 1));
        rows.alloc((size_t)blocks * p.rows_slab);
        p.rows_global = rows.p;
      }
      pairs.alloc(nnz / PAIR_ITEM + nnz / p.dmax + 1);
      smem = std::max(smem, (size_t)count_team_words(K, p.dmax, rows_in_smem) * 4);
      smem = std::max({smem, (size_t)WARPS * ORDER_WORDS<unsigned long long> * 4, (size_t)SEGMENT / 8});
      p.rel = rel.p;
      p.key = key.p;
      p.cin = cin.p;
      p.later = later.p;
      p.dplus = dplus.p;
      p.queue = queue.p;
      p.pairs = pairs.p;
      p.dag.doff = dag.off.p;
      p.dag.dadj = dag.adj.p;
      p.dag.outdeg = dag.outdeg.p;
      p.dag.heavy = dag.heavy;
    }
    if (m) {
      void *kern = k == 2 ? (void *)k_core<2> : k == 3 ? (void *)k_core<3> : k == 4 ? (void *)k_core<4>
                 : k == 5 ? (void *)k_core<5> : (void *)k_core<0>;
      // (raised to the most any launch uses, never lowered under another thread's launch)
      cudaFuncAttributes fa;
      CDS_CUDA(cudaFuncGetAttributes(&fa, kern));
      const size_t dyn_max = c->smem_optin - fa.sharedSizeBytes;
      if (smem > dyn_max) fail(CDS_ERR_CUDA, "peel team does not fit in shared memory");
      CDS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_max));
      int per_sm = 0;
      CDS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, smem));
      if (per_sm < 1) fail(CDS_ERR_CUDA, "peel kernel does not fit on an SM");
      blocks = std::min<unsigned>(blocks, coop_grid(c, std::min(per_sm, 2)));
      void *args[] = {&p};
      {
        ProfScope ps(c, s, "peel");
        CDS_CUDA(cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(THREADS), args, smem, s));
      }
      count_launch();
      CDS_CUDA(cudaGetLastError());
    }
  }
  if (k == 2) {
    k_edge_roots<<<c->sm_count * 8, 256, 0, s>>>(off, adj, out.core.p, n, R.p);
    count_launch();
  }
  // per-instance largest core (sizes the histograms), read with the status
  DBuf<uint32_t> imax(c, s, ninst);
  imax.zero();
  k_inst_maxcore<<<c->sm_count * 4, 256, 0, s>>>(out.core.p, n, of_vertex, imax.p);
  count_launch();
  uint32_t e = 0;
  {
    HostReads r(s);
    r.add(out.inst_max_core.data(), imax.p, ninst);
    r.add(&e, ctl_err);
    r.wait();
  }
  if (e & DEV_ERR_TIMEOUT) fail(CDS_ERR_TIMEOUT, "peel: device iteration budget exhausted");
  if (e) fail(CDS_ERR_CUDA, "peel: device error");
  std::vector<uint64_t> hoff(ninst + 1, 0);
  for (uint32_t i = 0; i < ninst; i++) {
    hoff[i + 1] = hoff[i] + out.inst_max_core[i] + 1;
    out.max_core = std::max(out.max_core, out.inst_max_core[i]);
  }
  DBuf<uint64_t> d_hoff(c, s, ninst + 1);
  DBuf<unsigned long long> hv(c, s, hoff[ninst]), hc(c, s, hoff[ninst]);
  DBuf<unsigned long long> bnum(c, s, ninst), bden(c, s, ninst);
  DBuf<uint32_t> ilev(c, s, ninst), blev(c, s, ninst);
  CDS_CUDA(cudaMemcpyAsync(d_hoff.p, hoff.data(), (ninst + 1) * 8, cudaMemcpyHostToDevice, s));
  hv.zero();
  hc.zero();
  {
    ProfScope ps(c, s, "peel_levels");
    const uint64_t bins = hoff[ninst], kept = std::min<uint64_t>(bins, n);
    const bool thin = bins > LEVELS_DIRECT && 12 * bins <= c->budget / 8;  // (of scratch)
    DBuf<uint32_t> used(c, s, thin ? bins : 0), lvl(c, s, thin ? kept : 0);
    DBuf<uint64_t> pos(c, s, thin ? bins + 1 : 0), off2(c, s, thin ? ninst + 1 : 0);
    DBuf<unsigned long long> v2(c, s, thin ? kept : 0), c2(c, s, thin ? kept : 0);
    used.zero();
    k_core_hist<<<c->sm_count * 4, 256, 0, s>>>(out.core.p, R.p, n, of_vertex, d_hoff.p, hv.p, hc.p, used.p);
    if (thin) {
      scan_u32(used.p, pos.p, bins, c, s);
      k_levels_in_use<<<c->sm_count * 8, 256, 0, s>>>(used.p, pos.p, bins, d_hoff.p, ninst, hv.p, hc.p, off2.p, v2.p,
                                                      c2.p, lvl.p);
      count_launch();
    }
    k_best_level<<<std::min<uint32_t>(ninst, c->sm_count * 4), 512, 0, s>>>(
        thin ? off2.p : d_hoff.p, thin ? v2.p : hv.p, thin ? c2.p : hc.p, lvl.p, ninst, bnum.p, bden.p, ilev.p,
        blev.p);
    count_launch(2);
  }
  CDS_CUDA(cudaGetLastError());
  std::vector<unsigned long long> hn(ninst), hd(ninst);
  uint32_t sweeps = 0;
  {
    HostReads r(s);
    r.add(hn.data(), bnum.p, ninst);
    r.add(hd.data(), bden.p, ninst);
    r.add(out.inst_levels.data(), ilev.p, ninst);
    r.add(out.best_level.data(), blev.p, ninst);
    r.add(&sweeps, ctl_sweeps);
    r.wait();
  }
  if (c->prof) {
    unsigned long long hph[3];
    {
      HostReads r(s);
      r.add(hph, phase.p, 3);
      r.wait();
    }
    std::lock_guard<std::mutex> g(c->mu);
    auto &slot = c->prof_done["peel_sweeps"];
    slot.first += 1;
    slot.second += sweeps;
    static const char *pn[3] = {"peel_phase_order", "peel_phase_count", "peel_phase_lower"};
    for (int i = 0; i < 3; i++) {
      auto &a = c->prof_done[pn[i]];
      a.first += 1;
      a.second += hph[i] / 1e6;
    }
  }
  for (uint32_t i = 0; i < ninst; i++) {
    out.best_num[i] = hn[i];
    out.best_den[i] = hd[i];
    out.levels = std::max(out.levels, out.inst_levels[i]);
  }
}

}  // namespace cds
