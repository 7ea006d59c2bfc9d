// list_kernels.cuh -- device code of the k-clique listing (see listing.cu
// for the method).  Included by every translation unit that launches it.
#pragma once
#include "device_util.cuh"
#include "dag_kernels.cuh"
#include "cds.h"

#include <type_traits>

namespace {

constexpr int WARP_DMAX = 128;    // out-degree limit of a warp team
constexpr int BLOCK_DMAX = 1024;  // out-degree limit for rows in shared memory
constexpr int DFS_WMAX = 32;      // bitmap words a DFS mask may need (k >= 5)

struct ListParams {
  const uint64_t *doff;
  const uint32_t *dadj;
  const uint32_t *outdeg;
  const uint32_t *deg;             // undirected degree
  const uint32_t *roots;
  const uint32_t *nroots;          // root count, on the device
  uint32_t *work;                  // dynamic scheduling cursor
  uint32_t *cdeg;                  // pass 1: clique degree (atomic), when cdeg64 is null
  unsigned long long *cdeg64;      // pass 1: clique degree as u64 (no 2^32 cap)
  unsigned long long *root_cnt;    // pass 1: cliques per root vertex
  const unsigned long long *base;  // pass 2: first clique index per vertex
  uint32_t *out;                   // pass 2: clique records
  uint32_t dmax;                   // team capacity (entries)
  uint32_t team_words;             // shared-memory words per team
  HeavyBits heavy;                 // adjacency among the heavy vertices
  uint32_t *rows_global;           // block teams: rows outside shared memory
  uint64_t rows_slab;              // words per block slab
  uint32_t *err;
  uint32_t k;                      // clique size (used by the generic k >= 5 path)
};

template <bool TB>
struct Team {
  __device__ __forceinline__ static int size() { return TB ? (int)blockDim.x : 32; }
  __device__ __forceinline__ static int rank() { return TB ? (int)threadIdx.x : (int)lane_id(); }
  __device__ __forceinline__ static int warps() { return TB ? (int)(blockDim.x >> 5) : 1; }
  __device__ __forceinline__ static int warp() { return TB ? (int)(threadIdx.x >> 5) : 0; }
  __device__ __forceinline__ static bool any(bool x) {  // over the team, which it synchronises
    if (TB) return __syncthreads_or(x) != 0;
    const bool r = __any_sync(CDS_FULL, x);
    __syncwarp();
    return r;
  }
  __device__ __forceinline__ static void sync() {
    if (TB) __syncthreads();
    else __syncwarp();
  }
  // exclusive scan of one value per team thread; *tot = team total
  template <class T>
  __device__ __forceinline__ static T scan(T v, T *tot) {
    if (TB) return block_exclusive_scan<T>(v, tot);
    T inc = warp_inclusive_scan(v);
    *tot = __shfl_sync(CDS_FULL, inc, 31);
    return inc - v;
  }
  template <class T>
  __device__ __forceinline__ static T sum(T v) {
    T tot;
    scan<T>(v, &tot);
    return tot;
  }
};

// first index i with P[i+1] > p, for P ascending with P[0] = 0
__device__ __forceinline__ uint32_t find_row(const uint32_t *P, uint32_t d, uint32_t p) {
  uint32_t lo = 0, hi = d;  // answer in [0, d)
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (P[mid] <= p) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ uint32_t nth_in_row(const uint32_t *row, uint32_t r) {
  for (uint32_t w = 0;; w++) {
    const uint32_t c = __popc(row[w]);
    if (r < c) return (w << 5) + (uint32_t)select_bit(row[w], (int)r);
    r -= c;
  }
}

template <int K>
struct CountOf {
  using type = uint32_t;  // a local count times k-2 stays below 2^32 (at most 1,024 local vertices at k = 5)
};
template <>
struct CountOf<0> {
  using type = unsigned long long;
};

// The local graph of a sorted vertex set A[0..d): hit(i, j) for every DAG arc
// A[i] -> A[j] whose tail is light.  (Arcs between heavy vertices are in the
// adjacency bitmap of the heavy vertices, and every arc out of a heavy vertex
// ends in one: arcs climb in degree.)  A warp takes a group of up to 32 rows and
// walks their out-lists laid end to end (a prefix over their lengths in
// registers), two steps of 32 entries in flight; light lists are short, and a
// step per list would leave most lanes idle and wait for three dependent loads
// (vertex, offset, entry) per row.  Team-wide; the caller synchronises after.
constexpr uint32_t LIGHT = 0xFFFFFFFFu;  // no heavy id
template <bool TB, class Hit>
__device__ __forceinline__ void light_arcs(const uint32_t *A, const uint32_t *hid, uint32_t d,
                                           const uint64_t *__restrict__ doff, const uint32_t *__restrict__ dadj,
                                           const uint32_t *__restrict__ outdeg, Hit hit) {
  constexpr int U = 2;
  const uint32_t lane = lane_id(), nw = Team<TB>::warps();
  uint32_t g = (d + nw - 1) / nw;
  g = g > 32 ? 32 : g;
  const uint32_t lo_id = A[0], hi_id = A[d - 1];
  for (uint32_t r0 = Team<TB>::warp() * g; r0 < d; r0 += nw * g) {
    const uint32_t n = min(g, d - r0);
    uint32_t len = 0;
    const uint32_t *list = nullptr;
    if (lane < n && hid[r0 + lane] == LIGHT) {
      const uint32_t a = A[r0 + lane];
      len = outdeg[a];
      list = dadj + doff[a];
    }
    const uint32_t incl = warp_inclusive_scan(len), ex = incl - len;
    const uint32_t total = __shfl_sync(CDS_FULL, incl, 31);
    for (uint32_t f0 = 0; f0 < total; f0 += 32 * U) {
      uint32_t r[U], b[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const uint32_t f = f0 + 32u * u + lane;
        r[u] = 0;
#pragma unroll
        for (uint32_t s = 16; s > 0; s >>= 1) {  // the last row that starts at or before f
          const uint32_t e = __shfl_sync(CDS_FULL, ex, (r[u] + s) & 31u);
          if (r[u] + s < n && e <= f) r[u] += s;
        }
        const uint32_t *p = reinterpret_cast<const uint32_t *>(
            __shfl_sync(CDS_FULL, reinterpret_cast<unsigned long long>(list), r[u]));
        const uint32_t at = f - __shfl_sync(CDS_FULL, ex, r[u]);
        b[u] = f < total ? p[at] : 0xFFFFFFFFu;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (b[u] < lo_id || b[u] > hi_id) continue;
        uint32_t lo = 0, hi = d;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (A[mid] < b[u]) lo = mid + 1;
          else hi = mid;
        }
        if (lo < d && A[lo] == b[u]) hit(r0 + r[u], lo);
      }
    }
  }
}

// Heavy part of the local graph: one word at a time of each row, word(i, w, m)
// with bit l of m set when A[i] and A[32 w + l] are adjacent heavy vertices.  A
// lane reads the bit of its column from row i of the heavy bitmap and a ballot
// makes the word, so 32 pairs cost one load and no search or atomic.  Rows of
// fewer than four words are taken as one sequence with HEAVY_U loads in flight
// (each comes from L2); longer ones a row at a time, which saves instructions.
// Word-uniform calls, every word of every row once, a row's words in order (zero
// where nothing is heavy).  Returns whether the calling warp met a light vertex.
constexpr int HEAVY_U = 8;
template <bool TB, class Word>
__device__ __forceinline__ bool heavy_words(const HeavyBits &hb, const uint32_t *hid, uint32_t d, Word word) {
  const uint32_t lane = lane_id(), W = (d + 31) >> 5, step = Team<TB>::warps();
  bool light = false;
  uint32_t i = Team<TB>::warp(), w = 0;
  if (W >= 4) {
    for (; i < d; i += step) {
      const uint32_t hi = hid[i];
      light |= hi == LIGHT;
      const uint32_t *row = hb.bits + (size_t)hi * hb.words;
#pragma unroll 4
      for (w = 0; w < W; w++) {
        const uint32_t j = w * 32 + lane;
        const uint32_t hj = j < d && hi != LIGHT ? hid[j] : LIGHT;
        const bool on = hj != LIGHT && (row[hj >> 5] >> (hj & 31)) & 1u;
        word(i, w, __ballot_sync(CDS_FULL, on));
      }
    }
    return light;
  }
  while (i < d) {
    uint32_t x[HEAVY_U], row[HEAVY_U], at[HEAVY_U];
    bool on[HEAVY_U];
#pragma unroll
    for (int u = 0; u < HEAVY_U; u++) {
      row[u] = i;
      at[u] = w;
      x[u] = 0;
      on[u] = i < d;
      if (on[u]) {
        const uint32_t hi = hid[i], j = w * 32 + lane, hj = j < d ? hid[j] : LIGHT;
        light |= hi == LIGHT;
        if (hi != LIGHT && hj != LIGHT) x[u] = hb.bits[(size_t)hi * hb.words + (hj >> 5)] >> (hj & 31);
        if (++w == W) {
          w = 0;
          i += step;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < HEAVY_U; u++)
      if (on[u]) word(row[u], at[u], __ballot_sync(CDS_FULL, x[u] & 1u));
  }
  return light;
}

// Depth-first enumeration of the `depth`-cliques {l1 < l2 < ...} inside mask M
// from position `first` on, over symmetric rows; leaf(path, s) for each, with
// s = the vertices adjacent to all of the path inside M.  Only for k >= 6.
// A path goes on only where the vertices left can complete it and leave one more.
template <class Leaf>
__device__ void dfs_common(const uint32_t *rows, uint32_t rs, uint32_t W, const uint32_t *M, uint32_t first,
                           int depth, Leaf leaf) {
  uint32_t stack[CDS_MAX_K][DFS_WMAX];
  uint32_t path[CDS_MAX_K];
  uint32_t pos[CDS_MAX_K];
  for (uint32_t w = 0; w < W; w++) stack[0][w] = M[w];
  int lvl = 0;
  pos[0] = first;
  while (lvl >= 0) {
    uint32_t b = pos[lvl];
    uint32_t found = 0xFFFFFFFFu;
    while ((b >> 5) < W) {
      const uint32_t word = stack[lvl][b >> 5] & (0xFFFFFFFFu << (b & 31));
      if (word) { found = ((b >> 5) << 5) + (uint32_t)(__ffs(word) - 1); break; }
      b = ((b >> 5) + 1) << 5;
    }
    if (found == 0xFFFFFFFFu) { lvl--; continue; }
    pos[lvl] = found + 1;
    path[lvl] = found;
    const uint32_t *row = rows + found * rs;
    uint32_t c = 0;
    if (lvl + 1 == depth) {
      for (uint32_t w = 0; w < W; w++) c += __popc(stack[lvl][w] & row[w]);
      if (c) leaf(path, c);
      continue;
    }
    for (uint32_t w = 0; w < W; w++) {
      stack[lvl + 1][w] = stack[lvl][w] & row[w];
      c += __popc(stack[lvl + 1][w]);
    }
    if ((int)c >= depth - lvl) {
      lvl++;
      pos[lvl] = found + 1;
    }
  }
}

// The same in registers, for a path of D vertices over rows of two to four words (the
// second pair of words zero where there are two; later: the bits of M a path may take
// next).  Adds what it finds to the path's counts; returns the sum of s.
struct Bits128 {
  unsigned long long lo, hi;
  __device__ __forceinline__ uint32_t size() const { return __popcll(lo) + __popcll(hi); }
  __device__ __forceinline__ Bits128 operator&(const Bits128 &o) const { return {lo & o.lo, hi & o.hi}; }
};
__device__ __forceinline__ Bits128 row_bits(const uint32_t *row) {  // (16-byte rows, padded with zeros)
  const uint4 x = *reinterpret_cast<const uint4 *>(row);
  return {(unsigned long long)x.y << 32 | x.x, (unsigned long long)x.w << 32 | x.z};
}
template <int D, class C>
__device__ __forceinline__ uint32_t paths_common(const uint32_t *rows, uint32_t rs, Bits128 M, Bits128 later, C *cnt) {
  uint32_t sum = 0;
  while (later.lo | later.hi) {
    uint32_t l;
    if (later.lo) {
      l = __ffsll((long long)later.lo) - 1;
      later.lo &= later.lo - 1;
    } else {
      l = 64 + __ffsll((long long)later.hi) - 1;
      later.hi &= later.hi - 1;
    }
    const Bits128 row = row_bits(rows + l * rs), N = M & row;
    uint32_t s = N.size();
    if constexpr (D > 1) s = s >= D ? paths_common<D - 1>(rows, rs, N, later & row, cnt) : 0u;
    if (s) {
      atomicAdd(&cnt[l], C(s));
      sum += s;
    }
  }
  return sum;
}

// The same for wider rows: the words of the P rows of the pair and the path so far are
// read again at each step (a stack of masks would be in local memory).  Of 1,024 vertices
// paths of two sum up to 5.3e8, longer ones pass 32 bits.
template <int D>
using PathSum = std::conditional_t<(D > 2), unsigned long long, uint32_t>;
template <int P, int D, class C>
__device__ __forceinline__ PathSum<D> paths_wide(const uint32_t *rows, uint32_t rs, uint32_t W,
                                                 const uint32_t *(&r)[P], uint32_t from, C *cnt) {
  PathSum<D> sum = 0;
  static_assert(D <= 3, "a step's own sum is held in 32 bits");
  for (uint32_t w = from >> 5; w < W; w++) {
    uint32_t m = w == (from >> 5) ? 0xFFFFFFFFu << (from & 31) : 0xFFFFFFFFu;
#pragma unroll
    for (int x = 0; x < P; x++) m &= r[x][w];
    for (; m; m &= m - 1) {
      const uint32_t l = w * 32 + __ffs(m) - 1;
      const uint32_t *q[P + 1];
#pragma unroll
      for (int x = 0; x < P; x++) q[x] = r[x];
      q[P] = rows + l * rs;
      uint32_t s = 0;
      for (uint32_t y = 0; y < W; y += 4) {
        uint4 a = *reinterpret_cast<const uint4 *>(q[0] + y);
#pragma unroll
        for (int x = 1; x <= P; x++) {
          const uint4 b = *reinterpret_cast<const uint4 *>(q[x] + y);
          a.x &= b.x;
          a.y &= b.y;
          a.z &= b.z;
          a.w &= b.w;
        }
        s += __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);
      }
      if constexpr (D > 1) s = s >= D ? paths_wide<P + 1, D - 1>(rows, rs, W, q, l + 1, cnt) : 0u;
      if (s) {
        atomicAdd(&cnt[l], C(s));
        sum += s;
      }
    }
  }
  return sum;
}

// Cliques of S vertices of mask M, over symmetric rows of one word.
template <int S>
__device__ __forceinline__ uint32_t word_cliques(const uint32_t *rows, uint32_t M) {
  uint32_t total = 0;
  while (__popc(M) >= S) {
    const uint32_t l = __ffs(M) - 1;
    M &= M - 1;
    const uint32_t N = M & rows[l];
    if constexpr (S == 2) total += __popc(N);
    else total += word_cliques<S - 1>(rows, N);
  }
  return total;
}
// The same for a size (2 or more) that is not known when compiling.
__device__ __forceinline__ unsigned long long cliques_in_word(const uint32_t *rows, uint32_t M, int size) {
  uint32_t left[CDS_MAX_K];  // by members chosen: who may be the next
  unsigned long long total = 0;
  int l = 0;
  left[0] = M;
  for (;;) {
    const uint32_t m = left[l];
    if ((int)__popc(m) < size - l) {
      if (l-- == 0) return total;
      continue;
    }
    left[l] = m & (m - 1);
    const uint32_t next = left[l] & rows[__ffs(m) - 1];
    if (l + 2 == size) total += __popc(next);
    else left[++l] = next;
  }
}

// Words from one symmetric row to the next: a row of more than one word is
// padded with zeros to whole 16-byte pieces, an odd number of them apart, so that
// eight lanes reading a piece each of different rows meet different banks.
__host__ __device__ constexpr uint32_t row_stride(uint32_t W) { return W <= 1 ? 1u : 4u * (((W + 3) / 4) | 1u); }

// What a counting team keeps in shared memory: the local vertices, their
// heavy ids and counts (64-bit for the generic k >= 6) and, for k >= 4, the rows
// unless they live in global memory.
__host__ __device__ constexpr uint32_t count_team_words(int K, uint32_t dmax, bool rows_in_smem) {
  const uint32_t d4 = (dmax + 3) & ~3u;
  uint32_t words = d4 * (K == 0 ? 4 : 3);
  if (K != 3 && rows_in_smem) words += dmax * row_stride((dmax + 31) / 32);
  return (words + 3) & ~3u;
}
// bits common to two (three) rows
__device__ __forceinline__ uint32_t common(const uint32_t *a, const uint32_t *b, uint32_t W) {
  if (W == 1) return __popc(*a & *b);
  uint32_t s = 0;
  for (uint32_t w = 0; w < W; w += 4) {
    const uint4 x = *reinterpret_cast<const uint4 *>(a + w), y = *reinterpret_cast<const uint4 *>(b + w);
    s += __popc(x.x & y.x) + __popc(x.y & y.y) + __popc(x.z & y.z) + __popc(x.w & y.w);
  }
  return s;
}
__device__ __forceinline__ uint32_t common(const uint32_t *a, const uint32_t *b, const uint32_t *c, uint32_t W) {
  if (W == 1) return __popc(*a & *b & *c);
  uint32_t s = 0;
  for (uint32_t w = 0; w < W; w += 4) {
    const uint4 x = *reinterpret_cast<const uint4 *>(a + w), y = *reinterpret_cast<const uint4 *>(b + w),
                z = *reinterpret_cast<const uint4 *>(c + w);
    s += __popc(x.x & y.x & z.x) + __popc(x.y & y.y & z.y) + __popc(x.z & y.z & z.z) + __popc(x.w & y.w & z.w);
  }
  return s;
}

// A writing team: the local vertices and heavy ids, the prefix over the rows'
// popcounts, the rows.
// Its rows are an odd number of words apart: lanes reading different rows hit
// different banks.
__host__ __device__ constexpr uint32_t write_stride(uint32_t W) { return W | 1u; }
__host__ __device__ constexpr uint32_t write_team_words(uint32_t dmax, bool rows_in_smem) {
  const uint32_t d4 = (dmax + 3) & ~3u;
  return (3 * d4 + 4 + (rows_in_smem ? dmax * write_stride((dmax + 31) / 32) : 0u) + 3) & ~3u;
}

// Words of a block's rows in global memory (out-degrees past BLOCK_DMAX), a multiple
// of 16 bytes.  Both passes use the same slabs, each with its own stride, and neither
// stride is the larger one everywhere (36 words: 36 counting, 37 writing).
__host__ __device__ constexpr uint64_t rows_slab_words(uint32_t dmax) {
  const uint32_t W = (dmax + 31) / 32, a = row_stride(W), b = write_stride(W);
  return ((uint64_t)dmax * (a > b ? a : b) + 3) & ~(uint64_t)3;
}
// every root up to dmax fits: d rows, as far apart as for d vertices
constexpr bool slabs_hold_their_rows() {
  for (uint32_t dmax = 1025; dmax <= 8192; dmax++) {
    const uint32_t W = (dmax + 31) / 32;
    if (dmax * (uint64_t)row_stride(W) > rows_slab_words(dmax)) return false;
    if (dmax * (uint64_t)write_stride(W) > rows_slab_words(dmax)) return false;
    if (row_stride(W) < row_stride(W - 1) || write_stride(W) < write_stride(W - 1)) return false;  // (smaller d)
  }
  return true;
}
static_assert(slabs_hold_their_rows(), "rows in global memory leave their block's slab");

// The (k-1)-cliques of the local graph G[A]: cnt[i] = those that hold A[i],
// times k-2 (divided out by the caller), for K = 3, 4, 5 and any k (K = 0).
//
// Rows are symmetric (both directions of an arc), so a pair (i, j) of adjacent
// vertices with s = |row_i & row_j| adds s to both ends and every clique is met
// once per edge (k = 4), with no step per clique: the oriented rows this
// replaces found each clique once and then paid a shared-memory atomic for its
// last member.  For k = 5 the same with triangles i < j < l, for k >= 6 with the
// (k-2)-cliques of a search from each pair: by masks in registers for k = 6, 7 (rows of
// two to four words: all of the path's, wider ones: read again at each step), by a stack in
// local memory for larger k.  (Stack alone, a word's pairs to its lanes: R-MAT 8,192,
// edge factor 6, k = 6 counted in 1.31 ms and 0.82 this way, its core numbers
// in 7.6 and 4.8; a random graph of 1,200 vertices and degree 300 4.7 and 3.9, 73.7 and 29.5.)  k = 3 counts local degrees and needs
// no rows.  A warp takes a row and gives each word's 32 vertices to its lanes
// (where cliques are many the rows are dense: about two in three of the pairs at
// R-MAT scale 18, edge factor 16); neighbourhoods of at most 32 need one word a
// row and a lane each.  Bound by instruction issue (2.9 of 4 slots with the
// searched rows), so the step that counts is the row building: by binary
// search of every out-list 5.9 ms for the 2.29 G 4-cliques of that graph, by
// bitmap words and ballots 2.2 ms.
// ONE: d is at most 32.
template <int K, bool TB, class C, bool ONE = false>
__device__ void local_count(const uint32_t *A, uint32_t *hid, uint32_t d, const HeavyBits &hb,
                            const uint64_t *doff, const uint32_t *dadj, const uint32_t *outdeg, uint32_t *rows,
                            C *cnt, int kk) {
  using T = Team<TB>;
  const int tr = T::rank(), ts = T::size();
  const uint32_t lane = lane_id(), W = (d + 31) >> 5, rs = row_stride(W);
  bool light;
  if (K == 3) {
    uint32_t deg = 0;
    light = heavy_words<TB>(hb, hid, d, [&](uint32_t i, uint32_t w, uint32_t m) {
      deg = (w ? deg : 0u) + __popc(m);
      if (w + 1 == W && lane == 0) cnt[i] = deg;
    });
  } else {
    light = heavy_words<TB>(hb, hid, d, [&](uint32_t i, uint32_t w, uint32_t m) {
      if (lane == 0) rows[i * rs + w] = m;
    });
    const uint32_t pad = (rs == 1 ? 1u : (W + 3) & ~3u) - W;  // words read past the row's last
    for (uint32_t i = tr; i < d * pad; i += ts) rows[(i / pad) * rs + W + i % pad] = 0;
    for (uint32_t i = tr; i < d; i += ts) cnt[i] = 0;
  }
  if (T::any(light)) {  // synchronises the team
    light_arcs<TB>(A, hid, d, doff, dadj, outdeg, [&](uint32_t i, uint32_t j) {
      if (K == 3) {
        atomicAdd(&cnt[i], C(1));
        atomicAdd(&cnt[j], C(1));
      } else {
        atomicOr(&rows[i * rs + (j >> 5)], 1u << (j & 31));
        atomicOr(&rows[j * rs + (i >> 5)], 1u << (i & 31));
      }
    });
    T::sync();
  }
  if (K == 3) return;
  static_assert(!ONE || !TB, "a warp's");
  if (!TB && (ONE || W == 1)) {
    const uint32_t row = lane < d ? rows[lane * rs] : 0u;
    C s = 0;
    if (K == 4) {
      for (uint32_t j = 0; j < d; j++) {
        const uint32_t rj = __shfl_sync(CDS_FULL, row, j);
        if ((row >> j) & 1u) s += __popc(row & rj);
      }
    } else if (K == 0) {  // each lane the cliques among its own neighbours, no step shared and none atomic
      if (kk == 6) s = word_cliques<4>(rows, row);
      else if (kk == 7) s = word_cliques<5>(rows, row);
      else if (kk == 8) s = word_cliques<6>(rows, row);
      else s = cliques_in_word(rows, row, kk - 2);
      s *= (uint32_t)(kk - 2);
    } else {
      for (uint32_t m = row; m; m &= m - 1) {
        const uint32_t j = __ffs(m) - 1;
        const uint32_t mj = row & rows[j * rs] & ~((2u << j) - 1u);
        for (uint32_t q = mj; q; q &= q - 1) s += __popc(mj & rows[(__ffs(q) - 1) * rs]);
      }
      s = s / 2 * 3;  // each triangle of the row was met from two of its pairs' first ends
    }
    if (lane < d) cnt[lane] = s;
    T::sync();
    return;
  }
  if constexpr (ONE) return;
  if constexpr (K == 0) {
    // the pairs i < j, a thread each, by their number in a prefix over the rows: a
    // pair's search takes from nothing to many steps, and most of a word's lanes would
    // wait for the longest (the prefix lies where the heavy ids were)
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < d; i0 += ts) {
      const uint32_t i = i0 + tr;
      uint32_t n = 0, tot;
      if (i < d)
        for (uint32_t w = i >> 5; w < W; w++)
          n += __popc(rows[i * rs + w] & (w == (i >> 5) ? ~((2u << (i & 31)) - 1u) : 0xFFFFFFFFu));
      const uint32_t ex = T::template scan<uint32_t>(n, &tot);
      if (i < d) hid[i] = carry + ex;
      carry += tot;
    }
    T::sync();
    for (uint32_t q = tr; q < carry; q += ts) {
      const uint32_t i = find_row(hid, d, q);
      const uint32_t *ri = rows + i * rs;
      uint32_t r = q - hid[i], w0 = i >> 5, m = ri[w0] & ~((2u << (i & 31)) - 1u);
      for (; r >= (uint32_t)__popc(m); m = ri[++w0]) r -= __popc(m);
      const uint32_t j = w0 * 32 + (uint32_t)select_bit(m, (int)r);
      const uint32_t *rj = rows + j * rs;
      C sum = 0;
      if (W == 1 || kk > 7) {
        uint32_t M[DFS_WMAX];
        int both = 0;
        for (uint32_t w = 0; w < W; w++) {
          M[w] = ri[w] & rj[w];
          both += __popc(M[w]);
        }
        if (both < kk - 3) continue;
        dfs_common(rows, rs, W, M, j + 1, kk - 4, [&](const uint32_t *path, uint32_t s) {
          for (int t = 0; t < kk - 4; t++) atomicAdd(&cnt[path[t]], C(s));
          sum += s;
        });
      } else if (W <= 4) {
        const Bits128 M = row_bits(ri) & row_bits(rj);
        if ((int)M.size() < kk - 3) continue;
        const Bits128 later = M & Bits128{j < 63 ? ~0ull << (j + 1) : 0ull,
                                          j < 63 ? ~0ull : j < 127 ? ~0ull << (j - 63) : 0ull};
        if (kk == 5) sum = paths_common<1>(rows, rs, M, later, cnt);
        else if (kk == 6) sum = paths_common<2>(rows, rs, M, later, cnt);
        else sum = paths_common<3>(rows, rs, M, later, cnt);
      } else {
        if ((int)common(ri, rj, W) < kk - 3) continue;
        const uint32_t *pair[2] = {ri, rj};
        if (kk == 5) sum = paths_wide<2, 1>(rows, rs, W, pair, j + 1, cnt);
        else if (kk == 6) sum = paths_wide<2, 2>(rows, rs, W, pair, j + 1, cnt);
        else sum = paths_wide<2, 3>(rows, rs, W, pair, j + 1, cnt);
      }
      if (sum) {
        atomicAdd(&cnt[i], sum);
        atomicAdd(&cnt[j], sum);
      }
    }
  } else for (uint32_t i = T::warp(); i < d; i += T::warps()) {
    const uint32_t *ri = rows + i * rs;
    C mine = 0;
    for (uint32_t w0 = i >> 5; w0 < W; w0++) {
      uint32_t m = ri[w0];
      if (w0 == (i >> 5)) m &= ~((2u << (i & 31)) - 1u);  // neighbours after i
      if (!((m >> lane) & 1u)) continue;
      const uint32_t j = w0 * 32 + lane;
      const uint32_t *rj = rows + j * rs;
      C sum = 0;
      if (K == 4) {
        sum = common(ri, rj, W);
      } else {  // 5
        uint32_t all = 0;
        for (uint32_t w = w0; w < W; w++) {
          uint32_t m2 = ri[w] & rj[w];
          if (w == w0) m2 &= ~((2u << lane) - 1u);
          for (; m2; m2 &= m2 - 1) {
            const uint32_t l = (w << 5) + (uint32_t)(__ffs(m2) - 1);
            const uint32_t s = common(ri, rj, rows + l * rs, W);
            if (s) atomicAdd(&cnt[l], C(s));
            all += s;
          }
        }
        sum = all;
      }
      if (sum) atomicAdd(&cnt[j], sum);
      mine += sum;
    }
    mine = warp_sum(mine);
    if (lane == 0 && mine) atomicAdd(&cnt[i], mine);
  }
  T::sync();
}

// Pass 1: cliques of each root, and clique degrees.  Warp teams take roots of
// out-degree up to p.dmax, block teams larger ones.
template <int K, bool TB>
__global__ void k_count(ListParams p) {
  using T = Team<TB>;
  using C = typename CountOf<K>::type;
  const int KK = K ? K : (int)p.k;
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint32_t s_root;
  uint32_t *S = sm + (TB ? 0u : (threadIdx.x >> 5) * p.team_words);
  const uint32_t d4 = (p.dmax + 3) & ~3u;
  C *cnt = reinterpret_cast<C *>(S);
  uint32_t *A = S + d4 * (sizeof(C) / 4);
  uint32_t *hid = A + d4;
  uint32_t *rows = (TB && p.rows_global) ? p.rows_global + (uint64_t)blockIdx.x * p.rows_slab : hid + d4;
  const int tr = T::rank(), ts = T::size();
  const uint32_t nroots = *p.nroots;
  for (;;) {
    uint32_t r;
    if (TB) {
      if (threadIdx.x == 0) s_root = atomicAdd(p.work, 1u);
      __syncthreads();
      r = s_root;
      __syncthreads();
    } else {
      if (lane_id() == 0) r = atomicAdd(p.work, 1u);
      r = __shfl_sync(CDS_FULL, r, 0);
    }
    if (r >= nroots) break;
    const uint32_t u = p.roots[r];
    const uint32_t d = p.outdeg[u];
    const uint32_t W = (d + 31) >> 5;
    if ((K == 0 || K == 5) && W > (uint32_t)DFS_WMAX) {  // k >= 5 is limited to DFS_WMAX words
      if (tr == 0) atomicOr(p.err, DEV_ERR_OVERFLOW);
      continue;
    }
    if (d > p.dmax) {  // classification guarantees d <= dmax
      if (tr == 0) atomicOr(p.err, DEV_ERR_INTERNAL);
      continue;
    }
    const uint32_t *Au = p.dadj + p.doff[u];
    for (uint32_t i = tr; i < d; i += ts) {
      const uint32_t a = Au[i];
      A[i] = a;
      hid[i] = p.heavy.id(a);
    }
    T::sync();
    local_count<K, TB, C>(A, hid, d, p.heavy, p.doff, p.dadj, p.outdeg, rows, cnt, KK);
    unsigned long long mine = 0;
    for (uint32_t i = tr; i < d; i += ts) {
      const unsigned long long c = (unsigned long long)cnt[i] / (unsigned)(KK - 2);
      mine += c;
      if (c) {
        if (p.cdeg64) atomicAdd(&p.cdeg64[A[i]], c);
        else atomicAdd(&p.cdeg[A[i]], (uint32_t)c);
      }
    }
    const unsigned long long total = T::template sum<unsigned long long>(mine) / (unsigned)(KK - 1);
    if (tr == 0) {
      p.root_cnt[u] = total;
      if (total) {
        if (p.cdeg64) atomicAdd(&p.cdeg64[u], total);
        else atomicAdd(&p.cdeg[u], (uint32_t)total);
      }
    }
    T::sync();
  }
}

// Enumerates the (depth)-cliques inside mask M (W words) with DFS over the
// bitmap rows; calls leaf(path, depth) for each.  Only used for k >= 5.
template <class Leaf>
__device__ void dfs_cliques(const uint32_t *rows, uint32_t rs, uint32_t W, const uint32_t *M,
                            int depth, Leaf leaf) {
  uint32_t stack[CDS_MAX_K][DFS_WMAX];
  uint32_t path[CDS_MAX_K];
  uint32_t pos[CDS_MAX_K];
  for (uint32_t w = 0; w < W; w++) stack[0][w] = M[w];
  int lvl = 0;
  pos[0] = 0;
  while (lvl >= 0) {
    // next set bit of stack[lvl] at or after pos[lvl]
    uint32_t b = pos[lvl];
    uint32_t found = 0xFFFFFFFFu;
    while ((b >> 5) < W) {
      const uint32_t word = stack[lvl][b >> 5] & (0xFFFFFFFFu << (b & 31));
      if (word) { found = ((b >> 5) << 5) + (uint32_t)(__ffs(word) - 1); break; }
      b = ((b >> 5) + 1) << 5;
    }
    if (found == 0xFFFFFFFFu) { lvl--; continue; }
    pos[lvl] = found + 1;
    path[lvl] = found;
    if (lvl + 1 == depth) {
      leaf(path, depth);
      continue;
    }
    const uint32_t *row = rows + found * rs;
    uint32_t any = 0;
    for (uint32_t w = 0; w < W; w++) {
      stack[lvl + 1][w] = stack[lvl][w] & row[w];
      any |= stack[lvl + 1][w];
    }
    if (any) {
      lvl++;
      pos[lvl] = 0;
    }
  }
}

// Pass 2: clique records at each root's offset.  K = 3 and K = 4 are
// specialised; K = 0 is the generic path for k >= 5.
template <int K, bool TB>
__global__ void k_list_write(ListParams p) {
  using T = Team<TB>;
  const int KK = K ? K : (int)p.k;
  extern __shared__ __align__(16) uint32_t sm[];
  __shared__ uint32_t s_root;
  uint32_t *S = sm + (TB ? 0u : (threadIdx.x >> 5) * p.team_words);
  const uint32_t d4 = (p.dmax + 3) & ~3u;
  uint32_t *A = S;               // [dmax]
  uint32_t *P = A + d4;          // [dmax+1] row-popcount prefix
  uint32_t *hid = P + d4 + 4;
  uint32_t *rows = (TB && p.rows_global) ? p.rows_global + (uint64_t)blockIdx.x * p.rows_slab : hid + d4;
  const int tr = T::rank(), ts = T::size();
  const uint32_t nroots = *p.nroots;
  for (;;) {
    uint32_t r;
    if (TB) {
      if (threadIdx.x == 0) s_root = atomicAdd(p.work, 1u);
      __syncthreads();
      r = s_root;
      __syncthreads();
    } else {
      if (lane_id() == 0) r = atomicAdd(p.work, 1u);
      r = __shfl_sync(CDS_FULL, r, 0);
    }
    if (r >= nroots) break;
    const uint32_t u = p.roots[r];
    const unsigned long long b0 = p.base[u];
    if (p.base[u + 1] == b0) continue;  // no clique has this root
    const uint32_t d = p.outdeg[u];
    const uint32_t W = (d + 31) >> 5;
    if (K == 0 && W > (uint32_t)DFS_WMAX) {  // DFS masks are limited to DFS_WMAX words
      if (tr == 0) atomicOr(p.err, DEV_ERR_OVERFLOW);
      continue;
    }
    if (d > p.dmax) {  // classification guarantees d <= dmax
      if (tr == 0) atomicOr(p.err, DEV_ERR_INTERNAL);
      continue;
    }
    const uint32_t rs = write_stride(W);
    const uint32_t *Au = p.dadj + p.doff[u];
    for (uint32_t i = tr; i < d; i += ts) {
      const uint32_t a = Au[i];
      A[i] = a;
      hid[i] = p.heavy.id(a);
    }
    T::sync();
    // local adjacency bitmap, oriented (a record's members follow DAG arcs): of
    // an adjacent heavy pair the arc is the one that climbs in (degree, id)
    const bool light = heavy_words<TB>(p.heavy, hid, d, [&](uint32_t i, uint32_t w, uint32_t m) {
      const uint32_t j = w * 32 + lane_id();
      bool on = (m >> lane_id()) & 1u;
      if (on) on = above(p.deg[A[j]], A[j], p.deg[A[i]], A[i]);
      m = __ballot_sync(CDS_FULL, on);
      if (lane_id() == 0) rows[i * rs + w] = m;
    });
    if (T::any(light)) {
      light_arcs<TB>(A, hid, d, p.doff, p.dadj, p.outdeg, [&](uint32_t i, uint32_t j) {
        atomicOr(&rows[i * rs + (j >> 5)], 1u << (j & 31));
      });
      T::sync();
    }
    // P = exclusive prefix of row popcounts
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < d; i0 += ts) {
      const uint32_t i = i0 + tr;
      uint32_t v = 0;
      if (i < d)
        for (uint32_t w = 0; w < W; w++) v += __popc(rows[i * rs + w]);
      uint32_t tot;
      const uint32_t ex = T::template scan<uint32_t>(v, &tot);
      if (i < d) P[i] = carry + ex;
      carry += tot;
    }
    if (tr == 0) P[d] = carry;
    T::sync();
    const uint32_t npairs = carry;
    if (K == 3) {
      for (uint32_t q = tr; q < npairs; q += ts) {
        const uint32_t i = find_row(P, d, q);
        const uint32_t j = nth_in_row(rows + i * rs, q - P[i]);
        uint32_t *o = p.out + (b0 + q) * 3;
        o[0] = u;
        o[1] = A[i];
        o[2] = A[j];
      }
    } else {
      unsigned long long wcarry = b0;
      for (uint32_t q0 = 0; q0 < npairs; q0 += ts) {
        const uint32_t q = q0 + tr;
        uint32_t i = 0, j = 0;
        unsigned long long c = 0;
        uint32_t M[K == 4 ? 4 : DFS_WMAX];
        const bool small = (K == 4) && W <= 4;
        if (q < npairs) {
          i = find_row(P, d, q);
          j = nth_in_row(rows + i * rs, q - P[i]);
          const uint32_t *ri = rows + i * rs, *rj = rows + j * rs;
          if (K == 4) {
            if (small) {
              for (uint32_t w = 0; w < W; w++) {
                M[w] = ri[w] & rj[w];
                c += __popc(M[w]);
              }
            } else {
              for (uint32_t w = 0; w < W; w++) c += __popc(ri[w] & rj[w]);
            }
          } else {
            uint32_t any = 0;
            for (uint32_t w = 0; w < W; w++) {
              M[w] = ri[w] & rj[w];
              any |= M[w];
            }
            if (any)
              dfs_cliques(rows, rs, W, M, KK - 3,
                          [&](const uint32_t *, int) { c++; });
          }
        }
        unsigned long long tot;
        const unsigned long long ex = T::template scan<unsigned long long>(c, &tot);
        if (c) {
          unsigned long long o = wcarry + ex;
          const uint32_t ai = A[i], aj = A[j];
          if (K == 4) {
            // a record that starts a 32-byte sector waits for its successor,
            // and the two go out as one 32-byte store (a whole sector)
            // instead of two half-sector stores
            const uint32_t *ri = rows + i * rs, *rj = rows + j * rs;
            uint4 pend = make_uint4(0u, 0u, 0u, 0u);
            bool has = false;
            for (uint32_t w = 0; w < W; w++) {
              uint32_t m = small ? M[w] : (ri[w] & rj[w]);
              while (m) {
                const uint32_t l = (w << 5) + (uint32_t)(__ffs(m) - 1);
                m &= m - 1;
                const uint4 r = make_uint4(u, ai, aj, A[l]);
                if (has) {
                  store_sector(p.out + (o - 1) * 4, pend, r);
                  has = false;
                } else if ((reinterpret_cast<uintptr_t>(p.out + o * 4) & 31u) == 0) {
                  pend = r;
                  has = true;
                } else {
                  *reinterpret_cast<uint4 *>(p.out + o * 4) = r;
                }
                o++;
              }
            }
            if (has) *reinterpret_cast<uint4 *>(p.out + (o - 1) * 4) = pend;
          } else {
            dfs_cliques(rows, rs, W, M, KK - 3, [&](const uint32_t *path, int depth) {
              uint32_t *rec = p.out + o * (unsigned long long)KK;
              rec[0] = u;
              rec[1] = ai;
              rec[2] = aj;
              for (int t = 0; t < depth; t++) rec[3 + t] = A[path[t]];
              o++;
            });
          }
        }
        wcarry += tot;
      }
    }
    T::sync();
  }
}

// roots with out-degree >= k-1, split by team size
__global__ void k_classify(const uint32_t *__restrict__ outdeg, uint32_t n, uint32_t kmin,
                           uint32_t warp_dmax, uint32_t *wl, uint32_t *wn, uint32_t *bl,
                           uint32_t *bn) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t d = outdeg[v];
    if (d < kmin) continue;
    if (d <= warp_dmax) wl[atomicAdd(wn, 1u)] = v;
    else bl[atomicAdd(bn, 1u)] = v;
  }
}

}  // namespace
