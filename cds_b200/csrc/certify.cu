// certify.cu -- proves that no subset of a component is denser than a given
// density, without a flow network.
//
// No counterpart in the reference, which runs max-flows until the search on alpha
// closes (cudaCode/main.cu:519-863); this is the dual of the same linear
// program.  Split every clique's k units among its members in any way and let
// load(v) be what v gets.  A set S of density p'/q' receives at least the k units
// of each clique inside it, so k |Psi(S)| <= sum over S of load(v), and with
// alpha = p/q and E = sum of max(0, load(v) - k alpha),
//     q |Psi(S)| - p |S| <= q E / k .
// The left side is an integer: E < k / q proves that no S is denser than alpha.
// When the whole component is the densest set of itself, equal loads exist, and
// they are found here by balancing weights: w(v) gives member v of a clique the
// share a = w(v) / sum of the clique's weights, and log w moves by the log of target
// / load over the load's own logarithmic derivative (1 - sum a^2 / sum a: Newton's
// step on the diagonal; without it vertices that need nearly all of their cliques
// approach that like 1/t), accelerated by Anderson's method over the last HIST
// differences (D. G. Anderson, "Iterative procedures for nonlinear integral
// equations", J. ACM 12, 1965).  5 to 16 passes over the cliques reach the bound on
// most R-MAT and planted graphs tried, 20 to 40 where levels split late (7 to 36
// and more without the derivative).
//
// A component that some subset S of it is denser than does not balance, and shows it
// by the eighth pass.  Its vertices by falling weight are then an order to take them
// away in (those that want more than their cliques hold go first): a pass counts
// every clique at its first vertex of that order, which gives the density of every
// remainder, and the densest one is S.  From there on S and the rest balance as two
// levels: the rest's weights are scaled up until cliques that cross give S nothing
// that counts, S aims at its own density and the rest at what is left.  E against
// the density of S proves it the densest, and when every other vertex stays below
// k alpha by more than E, no densest set holds one: S is the maximal one.  What
// does not balance after that goes to the flows, with S to start from.
//
// A pass never stores a clique.  The component's covered pairs are a symmetric
// bitmap of its vertices in shared memory; a warp takes a clique of k-2 vertices
// (none for k = 2, a vertex for k = 3, an edge for k = 4), deals the later common
// neighbours j to its lanes, and goes through that mask's members l together: lane j
// adds 1 / (sum of weights) where its row has l.  Every clique is so met twice, from j
// and from l, and each lane's sum belongs to its own j: met once, the sums of the last
// members need an atomic or a reduction per prefix, which cost five times the
// arithmetic saved.  Bound by instruction issue (64 % active at 746 vertices, k = 3).
// (Each lane walking the bits of its own row wastes no step, but
// finding a bit takes two operations of the unit that has the reciprocals, at a
// quarter of the rate: 33.6 ms for the nine passes of 1.14 G 4-cliques, 29.3 with one
// such operation, 23.8 this way.)  The proof itself
// is in integers: a last pass splits k 2^s units of every clique exactly, and the
// host checks E (and that the loads add up to every clique's units) in 128 bits.
//
// Measured against network build, warm split and push-relabel: 40 vertices and 1,499
// triangles 0.39 -> 0.14 ms, 470 vertices and 25,761 edges 0.69 -> 0.25, 112 and
// 1.18 M 4-cliques 1.5 -> 0.38, 746 and 9.3 M triangles 4.4 -> 1.3, 988 and 1.14 G
// 4-cliques 295 -> 31 with nine passes and the integer one (another seed's 1.15 G 36 to
// 37 with ten), and 62 GB of records and lists that are not built.
#include "core_rows.cuh"
#include "device_util.cuh"
#include "stages.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

namespace {

constexpr uint32_t MAX_N = 1024;   // vertices of a component: a word of a row per lane
constexpr int THREADS = 1024, WARPS = THREADS / 32;
constexpr uint32_t PARTS = 4;      // of the work, a block, with several components
constexpr int HIST = 8;            // differences Anderson's method combines
constexpr uint32_t MAX_PASSES = 48, MAX_ORDERS = 5;
constexpr uint64_t MAX_CLIQUES = 0xFFFFFFFFull;  // (counts at first vertices are 32-bit)
constexpr uint32_t ITEM_WORDS = 2; // k <= 3: words of l an item walks

struct Comp {
  uint32_t vbeg, n;       // local vertices
  uint32_t W, row;        // words a row (odd: lanes on different rows meet different banks), first word
  uint32_t item, nitems;  // its items (k = 4, 5: edges, from `item` on, ...
  uint32_t split;         // ... each split this many ways)
};
// The search's state of a component.
struct Level {
  double target[2];       // load to balance to: at the level of S (all, at first), of the rest
  double cap;             // k alpha
  double stop;            // E below this counts as reached
  unsigned long long psi; // cliques of S ...
  uint32_t size;          // ... and its vertices (0: none denser than asked was found)
  uint32_t since;         // pass the present levels began at
  uint32_t orders, split; // orders counted so far; whether one gave two levels
  unsigned long long p, q;  // alpha
};
struct Part {             // a piece of a component's items
  uint32_t comp, part, parts;
};

struct CertParams {
  uint32_t k, ncomp, nv;
  const Comp *comp;
  const uint32_t *rows;       // symmetric bitmap rows
  const uint32_t *item_u;     // k = 4, 5: the edges u < i by component (indexes in it)
  const uint32_t *item_i;
  const Part *part;           // [nparts] by component
  uint32_t nparts;
  Level *level;               // [ncomp]
  uint32_t *rest;             // [nv] 1: not in S
  uint32_t *rank;             // [nv] place in the order of falling weight
  uint32_t *first;            // [nv] cliques counted at each vertex
  uint32_t *wide;             // [ncomp] sums in double precision from now on
  uint32_t *state;            // [ncomp] BALANCE ... NOT_ASKED
  double *w;                  // [nv]
  double *T;                  // [nv] sum of 1 / (clique's weights) over the vertex's cliques
  float *T2;                  // [nv] the same of the squares
  unsigned long long *load;   // [2 nv] integer loads: low 32-bit halves, high halves summed
  double *X, *F;              // [(HIST+1) * nv] log-weights and residuals of the last passes
  double *G;                  // [ncomp * HIST * HIST] products of residual differences
  uint32_t *ctl;              // by pass mod 3: active components, parts taken (sums, firsts); [9]: shares
  GridBarrier *bar;
  uint32_t *err;
  unsigned long long spin_limit;
  uint32_t *passes;
  unsigned long long *phase_ns;  // [3] block 0's time in passes, updates, the integer pass (profiling; null: off)
};
enum : uint32_t { BALANCE = 0, REACHED = 1, GIVEN_UP = 2, COUNT = 3, NOT_ASKED = 4 };
// Log of the weights' ratio between the levels, at least: a clique that crosses gives the
// members of S at most e^-28 = 7e-13 of its units a member of the rest, so that 10^9 such
// cliques stay below a thousandth of one clique, and weights down to the floor
// of e^-60 keep their shares.
constexpr double LEVEL_GAP = 28.0;
constexpr int UNIT_BITS = 46;  // a clique has k 2^46 units

// Shared memory of a block: the component it works on.
struct Shared {
  uint32_t *rows;
  double *w, *acc;
  float *wf, *acc2;
};
__host__ __device__ constexpr size_t shared_bytes(uint32_t n, uint32_t W) {
  return (size_t)n * 24 + (size_t)n * W * 4 + 16;
}

__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1/d from the approximate single-precision reciprocal of d and one Newton step:
// relative error below 1e-13
__device__ __forceinline__ double newton(double d, float y0) {
  const double y = (double)y0;
  return y * fma(-d, y, 2.0);
}

// The j of a step: lane q of the warp takes the (q0 + q)-th bit of jmask (lane x
// holds word x; incl: the inclusive prefix of its popcounts).
__device__ __forceinline__ uint32_t deal(uint32_t jmask, uint32_t incl, uint32_t q) {
  uint32_t x = 0;  // the word that holds the q-th bit: the first with incl > q
#pragma unroll
  for (uint32_t st = 16; st > 0; st >>= 1) {
    const uint32_t e = __shfl_sync(CDS_FULL, incl, x + st - 1);
    if (e <= q) x += st;
  }
  const uint32_t xs = min(x, 31u), mw = __shfl_sync(CDS_FULL, jmask, xs);
  const uint32_t before = __shfl_sync(CDS_FULL, incl - __popc(jmask), xs);
  return xs * 32 + select_bit(mw, (int)(q - before));
}

// The pairs of adjacent vertices j in jmask and l in mask (lane x holds word x),
// each with the prefix one clique.  base: the prefix's weights.  Adds to every j's
// accumulators (the sum, and in single precision the sum of its squared shares) and
// returns this lane's sums over its j (every clique twice over the calls that cover
// all j; squares: relative to j's weight), over words [y0, y1) of mask; of the steps of 32 j every
// split-th from g on.  Two words at a time, a visit from each in flight.  WIDE:
// double precision; else single-precision terms, summed in double per j.
template <bool WIDE, int NP>
__device__ __forceinline__ double pair_sums(const Shared &sh, uint32_t y0, uint32_t y1, uint32_t W, uint32_t jmask,
                                            uint32_t mask, uint32_t g, uint32_t split, double base, const float *wp,
                                            float *squares) {
  const uint32_t lane = lane_id(), incl = warp_inclusive_scan((uint32_t)__popc(jmask));
  const uint32_t total = __shfl_sync(CDS_FULL, incl, 31);
  double tot = 0.0;
  for (uint32_t q0 = 32 * g; q0 < total; q0 += 32 * split) {
    const uint32_t jq = deal(jmask, incl, min(q0 + lane, total - 1));
    const bool on = q0 + lane < total;
    const uint32_t *row = sh.rows + jq * W;
    const double bj = base + sh.w[jq];
    const float bf = (float)bj, wj = sh.wf[jq];
    double s = 0.0, s2 = 0.0;
    float f = 0.0f, f2 = 0.0f, sq = 0.0f;
    for (uint32_t y = y0; y < y1; y++) {
      uint32_t m = __reduce_or_sync(CDS_FULL, lane == y ? mask : 0u);
      if (!m) continue;
      const uint32_t r = on ? row[y] : 0u;
      const float *wf = sh.wf + y * 32;
      const double *w = sh.w + y * 32;
#pragma unroll
      for (uint32_t b = 0; b < 32; b++) {
        if (!((m >> b) & 1u)) continue;  // (the whole warp)
        const float x = (r >> b) & 1u ? rcp(bf + wf[b]) : 0.0f;  // (0 for an absent one)
        if (WIDE) (b & 1 ? s2 : s) += newton(bj + w[b], x);
        else (b & 1 ? f2 : f) += x;
        const float z = x * wj;  // shares: their squares stay in range
        sq = fmaf(z, z, sq);
      }
    }
    if (WIDE) s += s2;
    else s = (double)f + (double)f2;
    if (s != 0.0) {
      atomicAdd(sh.acc + jq, s);
      atomicAdd(sh.acc2 + jq, sq);
    }
    tot += s;
#pragma unroll
    for (int x = 0; x < NP; x++) {
      const float r = wp[x] / wj;
      squares[x] += sq * r * r;
    }
  }
  return tot;
}

// The same in units: each member's share of a clique rounded down, j's summed into
// its load; what j and l leave (counted from the smaller of the two) goes to the
// prefix's NP vertices by weight, the remainder to the first.  k = 2 has no
// prefix: the larger end takes what the smaller leaves.  Both visits of a clique
// compute the same shares: the sum of the weights is taken in one order.
template <int NP>
__device__ __forceinline__ void pair_shares(const Shared &sh, uint32_t y0, uint32_t y1, uint32_t W, uint32_t jmask,
                                            uint32_t mask, uint32_t g, uint32_t split, double base, uint32_t k,
                                            const uint32_t *pre, unsigned long long *lo, unsigned long long *hi) {
  const uint32_t lane = lane_id(), incl = warp_inclusive_scan((uint32_t)__popc(jmask));
  const uint32_t total = __shfl_sync(CDS_FULL, incl, 31);
  const unsigned long long all = (unsigned long long)k << UNIT_BITS;
  const double units = (double)all;
  unsigned long long rem = 0;
  auto give = [&](uint32_t v, unsigned long long a) {
    atomicAdd(lo + v, a & 0xFFFFFFFFull);
    atomicAdd(hi + v, a >> 32);
  };
  for (uint32_t q0 = 32 * g; q0 < total; q0 += 32 * split) {
    const bool on = q0 + lane < total;
    const uint32_t j = deal(jmask, incl, min(q0 + lane, total - 1));
    const uint32_t *row = sh.rows + j * W;
    const double wj = sh.w[j];
    unsigned long long sum = 0;
    for (uint32_t y = y0; y < y1; y++) {
      const uint32_t my = __shfl_sync(CDS_FULL, mask, y);
      if (!my) continue;
      for (uint32_t m = on ? my & row[y] : 0u; m;) {
        const uint32_t b = 31 - __clz(m), l = y * 32 + b;
        m ^= 1u << b;
        const double wl = sh.w[l], d = base + (wj + wl), inv = newton(d, rcp((float)d));
        unsigned long long a = (unsigned long long)(units * ((j < l ? wj : wl) * inv));  // the smaller one's
        a = a < all ? a : all;
        unsigned long long c = all - a;  // and the larger one's
        if (NP > 0) {
          const unsigned long long z = (unsigned long long)(units * ((j < l ? wl : wj) * inv));
          c = z < c ? z : c;
        }
        sum += j < l ? a : c;
        if (j < l) rem += all - a - c;
      }
    }
    if (sum) give(j, sum);
    // a step adds at most 1,024 cliques of k 2^46 units to a lane: given before 32
    // lanes' sums could pass 64 bits
    if (NP > 0 && (q0 + 32 * split >= total || __any_sync(CDS_FULL, rem >> 56))) {
      const unsigned long long sum_rem = warp_sum(rem);
      rem = 0;
      if (lane == 0 && sum_rem) {
        unsigned long long left = sum_rem;
#pragma unroll
        for (int x = 1; x < NP; x++) {
          unsigned long long a = (unsigned long long)((double)sum_rem * (sh.w[pre[x]] / base));
          a = a < left ? a : left;
          left -= a;
          give(pre[x], a);
        }
        if (left) give(pre[0], left);
      }
    }
  }
}

// Every clique (once: l after j) counted at its member of smallest rank.
template <int NP>
__device__ __forceinline__ void pair_firsts(const Shared &sh, uint32_t y0, uint32_t y1, uint32_t W, uint32_t jmask,
                                            uint32_t mask, uint32_t g, uint32_t split, const uint32_t *pre) {
  const uint32_t lane = lane_id(), incl = warp_inclusive_scan((uint32_t)__popc(jmask));
  const uint32_t total = __shfl_sync(CDS_FULL, incl, 31);
  const uint32_t *rank = reinterpret_cast<const uint32_t *>(sh.wf);
  uint32_t *first = reinterpret_cast<uint32_t *>(sh.acc2);
  for (uint32_t q0 = 32 * g; q0 < total; q0 += 32 * split) {
    const bool on = q0 + lane < total;
    const uint32_t j = deal(jmask, incl, min(q0 + lane, total - 1));
    const uint32_t *row = sh.rows + j * W;
    uint32_t r0 = rank[j], v0 = j, n = 0;
#pragma unroll
    for (int x = 0; x < NP; x++)
      if (rank[pre[x]] < r0) {
        r0 = rank[pre[x]];
        v0 = pre[x];
      }
    for (uint32_t y = y0; y < y1; y++) {
      const uint32_t my = __shfl_sync(CDS_FULL, mask, y);
      if (!my) continue;
      uint32_t m = on && y >= (j >> 5) ? my & row[y] : 0u;
      if (y == (j >> 5)) m &= ~((2u << (j & 31)) - 1u);
      for (; m; m &= m - 1) {
        const uint32_t l = y * 32 + __ffs(m) - 1;
        if (rank[l] < r0) atomicAdd(first + l, 1u);
        else n++;
      }
    }
    if (n) atomicAdd(first + v0, n);
  }
}

// One pass over the components in the states of `want` (a bit each).  Blocks take
// parts from a counter (their list goes by component, so a block mostly stays with the
// one whose rows it has) and add their sums to the component's when they leave it.
enum Mode { SUMS, SHARES, FIRSTS };
template <int K, Mode MODE>
__device__ __noinline__ void pass_over(const CertParams &p, uint32_t want, uint32_t *take, uint32_t *loaded) {
  constexpr bool INT = MODE == SHARES;
  extern __shared__ __align__(16) char smem[];
  __shared__ uint32_t s_part, s_next;  // the block's next part, its warps' next item
  const uint32_t lane = lane_id();
  uint32_t cur = 0xFFFFFFFFu;
  Comp c{};
  // (derived from the array at each use: pointers that live across the loop lose
  // their address space, and every access then costs a generic one)
  auto areas = [&] {
    Shared sh;
    sh.w = reinterpret_cast<double *>(smem);
    sh.acc = sh.w + c.n;
    sh.wf = reinterpret_cast<float *>(sh.acc + c.n);
    sh.acc2 = sh.wf + c.n;
    sh.rows = reinterpret_cast<uint32_t *>(sh.acc2 + c.n);
    return sh;
  };
  auto leave = [&] {  // (every thread is past its items)
    if (cur == 0xFFFFFFFFu) return;
    const Shared sh = areas();
    if (MODE == FIRSTS)
      for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
        const uint32_t n = reinterpret_cast<uint32_t *>(sh.acc2)[v];
        if (n) atomicAdd(p.first + c.vbeg + v, n);
      }
    if (MODE == SUMS)
      for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x)
        if (sh.acc[v] != 0.0) {
          atomicAdd(p.T + c.vbeg + v, sh.acc[v]);
          atomicAdd(p.T2 + c.vbeg + v, sh.acc2[v]);
        }
    __syncthreads();
  };
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t x = atomicAdd(take, 1u);
      while (x < p.nparts && !((want >> __ldcg(p.state + p.part[x].comp)) & 1u)) x = atomicAdd(take, 1u);
      s_part = x;
      s_next = 0;
    }
    __syncthreads();
    if (s_part >= p.nparts) break;
    const Part pt = p.part[s_part];
    if (pt.comp != cur) {
      leave();
      cur = pt.comp;
      c = p.comp[cur];
      const Shared sh = areas();
      if (*loaded != cur)
        for (uint32_t i = threadIdx.x; i < c.n * c.W; i += blockDim.x) sh.rows[i] = p.rows[c.row + i];
      for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
        const double w = __ldcg(p.w + c.vbeg + v);
        sh.w[v] = w;
        sh.wf[v] = MODE == FIRSTS ? __uint_as_float(__ldcg(p.rank + c.vbeg + v)) : (float)w;
        sh.acc[v] = 0.0;
        sh.acc2[v] = 0.0f;  // (FIRSTS: a count of zero)
      }
      __syncthreads();
      if (threadIdx.x == 0) *loaded = cur;
    }
    const Shared sh = areas();
    auto row = [&](uint32_t v) { return lane < c.W ? sh.rows[v * c.W + lane] : 0u; };
    auto later = [&](uint32_t m, uint32_t v) {  // the bits of m past v
      const uint32_t w = v >> 5;
      return lane < w ? 0u : lane > w ? m : m & ~((2u << (v & 31)) - 1u);
    };
    unsigned long long *lo = p.load + c.vbeg, *hi = p.load + p.nv + c.vbeg;
    const bool wide = __ldcg(p.wide + pt.comp) != 0;
    // the pairs of one prefix, and what its own vertices get
    auto leaf = [&](uint32_t jmask, uint32_t mask, uint32_t y0, uint32_t y1, uint32_t g, uint32_t split, double base,
                    const uint32_t *pre) {
      if (!__any_sync(CDS_FULL, jmask)) return;
      if constexpr (MODE == FIRSTS) {
        pair_firsts<K - 2>(sh, y0, y1, c.W, jmask, mask, g, split, pre);
      } else if constexpr (INT) {
        pair_shares<K - 2>(sh, y0, y1, c.W, jmask, mask, g, split, base, p.k, pre, lo, hi);
      } else {
        constexpr int NP = K - 2;
        float wp[NP ? NP : 1], sq[NP ? NP : 1];
#pragma unroll
        for (int y = 0; y < NP; y++) {
          wp[y] = sh.wf[pre[y]];
          sq[y] = 0.0f;
        }
        const double t = wide ? pair_sums<true, NP>(sh, y0, y1, c.W, jmask, mask, g, split, base, wp, sq)
                              : pair_sums<false, NP>(sh, y0, y1, c.W, jmask, mask, g, split, base, wp, sq);
        const double h = 0.5 * warp_sum(t);
#pragma unroll
        for (int y = 0; y < NP; y++) {
          const float z = 0.5f * warp_sum(sq[y]);
          if (lane == 0) {
            atomicAdd(sh.acc + pre[y], h);
            atomicAdd(sh.acc2 + pre[y], z);
          }
        }
      }
    };
    // items are dealt to the parts in turn, and a part's to its warps as they come
    for (;;) {
      uint32_t it = 0;
      if (lane == 0) it = atomicAdd(&s_next, 1u);
      it = pt.part + pt.parts * __shfl_sync(CDS_FULL, it, 0);
      if (it >= c.nitems) break;
      if constexpr (K <= 3) {  // (vertex u for k = 3,) a word of j, a few words of l
        const uint32_t L = (c.W + ITEM_WORDS - 1) / ITEM_WORDS, jl = it % (c.W * L), u = it / (c.W * L);
        const uint32_t jw = jl / L, y0 = jl % L * ITEM_WORDS, y1 = min(y0 + ITEM_WORDS, c.W);
        const uint32_t pre[1] = {u};
        uint32_t mask;
        if constexpr (K == 2) mask = lane * 32 >= c.n ? 0u : 0xFFFFFFFFu >> (32 - min(32u, c.n - lane * 32));
        else mask = later(row(u), u);
        const bool some = __any_sync(CDS_FULL, lane >= y0 && lane < y1 && mask);
        if (some) leaf(lane == jw ? mask : 0u, mask, y0, y1, 0, 1, K == 2 ? 0.0 : sh.w[u], pre);
      } else {
        const uint32_t e = c.item + it / c.split, g = it % c.split, u = p.item_u[e], i = p.item_i[e];
        const uint32_t mask = later(row(u) & row(i), i);
        if constexpr (K == 4) {
          const uint32_t pre[2] = {u, i};
          leaf(mask, mask, i >> 5, c.W, g, c.split, sh.w[u] + sh.w[i], pre);
        } else {
          uint32_t turn = 0;
          for (uint32_t x2 = i >> 5; x2 < c.W; x2++)
            for (uint32_t m = __shfl_sync(CDS_FULL, mask, x2); m; m &= m - 1) {
              if (turn++ % c.split != g) continue;
              const uint32_t i2 = x2 * 32 + __ffs(m) - 1;
              const uint32_t pre[3] = {u, i, i2}, mask2 = later(mask & row(i2), i2);
              leaf(mask2, mask2, i2 >> 5, c.W, 0, 1, sh.w[u] + sh.w[i] + sh.w[i2], pre);
            }
        }
      }
    }
  }
  leave();
}

__device__ __forceinline__ double block_sum(double v, double *s) {
  v = warp_sum(v);
  if (lane_id() == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int x = 0; x < WARPS; x++) t += s[x];
  __syncthreads();
  return t;
}
__device__ __forceinline__ double block_max(double v, double *s) {
  v = warp_max(v);
  if (lane_id() == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = s[0];
  for (int x = 1; x < WARPS; x++) t = s[x] > t ? s[x] : t;
  __syncthreads();
  return t;
}

// The order of falling weight, for a count at each clique's first vertex.
__device__ __noinline__ void ask_order(const CertParams &p, uint32_t ci) {
  __shared__ double s_w[MAX_N];
  const Comp c = p.comp[ci];
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) s_w[v] = p.w[c.vbeg + v];
  __syncthreads();
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    uint32_t r = 0;
    for (uint32_t u = 0; u < c.n; u++) r += s_w[u] > s_w[v] || (s_w[u] == s_w[v] && u < v);
    p.rank[c.vbeg + v] = r;
    p.first[c.vbeg + v] = 0;
  }
  __syncthreads();
}

// After the count: the densest remainder of the order becomes S where it is denser
// than the present S (the component, at first).  Returns whether it is.
__device__ __noinline__ bool split_levels(const CertParams &p, uint32_t ci, uint32_t t, double *s) {
  __shared__ unsigned long long s_left[MAX_N];
  __shared__ uint32_t s_best;
  __shared__ uint32_t s_rank[MAX_N];
  const Comp c = p.comp[ci];
  Level &lv = p.level[ci];
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    s_rank[v] = p.rank[c.vbeg + v];
    s_left[s_rank[v]] = __ldcg(p.first + c.vbeg + v);
  }
  if (threadIdx.x == 0) s_best = 0xFFFFFFFFu;
  __syncthreads();
  // cliques left once the vertices of smaller rank are gone (a thread a rank)
  static_assert(MAX_N == THREADS, "a rank a thread");
  const uint32_t i = threadIdx.x;
  // (a scan of its own: with the 1,024 threads' block_exclusive_scan the kernel spills 8 bytes
  // more at k = 4, and the integer pass over 1.15 G 4-cliques takes 8.2 ms instead of 7.7)
  __shared__ unsigned long long s_warps[WARPS];
  static_assert(WARPS == 32, "a warp's sum a lane");
  const unsigned long long mine = i < c.n ? s_left[i] : 0ull, upto = warp_inclusive_scan(mine);
  if (lane_id() == 31) s_warps[i >> 5] = upto;
  __syncthreads();
  const unsigned long long sums = warp_inclusive_scan(s_warps[lane_id()]);
  const unsigned long long total = __shfl_sync(CDS_FULL, sums, 31), own = __shfl_sync(CDS_FULL, upto, 31);
  const unsigned long long gone = __shfl_sync(CDS_FULL, sums, i >> 5) - own + upto - mine;
  const unsigned long long left = total - gone;
  const double density = i < c.n ? (double)left / (double)(c.n - i) : -1.0;
  const double top = block_max(density, s);
  if (density == top) atomicMin(&s_best, i);
  __syncthreads();
  const uint32_t best = s_best;
  if (i == best) s_left[0] = left;
  __syncthreads();
  const unsigned long long psi = s_left[0];
  const uint32_t size = c.n - best;
  const double now = lv.target[0] / (double)p.k;  // density the top level aims at
  __syncthreads();
  if (best == 0 || !(top > now * (1.0 + 1e-12))) return false;
  if (threadIdx.x == 0) {
    // denser than alpha: the new alpha (in integers)
    const unsigned long long lh = __umul64hi(psi, lv.q), ll = psi * lv.q, rh = __umul64hi(lv.p, size), rl = lv.p * size;
    if (lh > rh || (lh == rh && ll > rl)) {
      unsigned long long a = psi, b = size;
      while (b) {
        const unsigned long long r = a % b;
        a = b;
        b = r;
      }
      lv.p = psi / a;
      lv.q = size / a;
      lv.psi = psi;
      lv.size = size;
      lv.cap = (double)p.k * (double)lv.p / (double)lv.q;
      lv.stop = 0.3 * (double)p.k / (double)lv.q;
    }
    lv.target[0] = (double)p.k * (double)psi / (double)size;
    lv.target[1] = (double)p.k * (double)(total - psi) / (double)best;
  }
  // the rest's weights above those of S by the gap
  double hi = -1e300, lo = 1e300;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    const double x = log(p.w[c.vbeg + v]);
    if (s_rank[v] < best) lo = x < lo ? x : lo;
    else hi = x > hi ? x : hi;
  }
  hi = block_max(hi, s);
  lo = -block_max(-lo, s);
  const double down = hi - lo + LEVEL_GAP;
  double mx = -1e300;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    const bool out = s_rank[v] < best;
    const double x = log(p.w[c.vbeg + v]) - (out || down < 0.0 ? 0.0 : down);
    p.X[(size_t)((t + 1) % (HIST + 1)) * p.nv + c.vbeg + v] = x;
    p.rest[c.vbeg + v] = out;
    mx = x > mx ? x : mx;
  }
  mx = block_max(mx, s);
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    const double d = p.X[(size_t)((t + 1) % (HIST + 1)) * p.nv + c.vbeg + v] - mx;
    p.w[c.vbeg + v] = exp(d < -60.0 ? -60.0 : d);
  }
  __syncthreads();
  return true;
}

// After pass t: the loads of component ci, and its next weights.  One block; the
// same block takes the component every time, so its history is its own.
__device__ __noinline__ void update(const CertParams &p, uint32_t ci, uint32_t t, uint32_t *active, double *s) {
  const Comp c = p.comp[ci];
  Level &lv = p.level[ci];
  if (__ldcg(p.state + ci) == COUNT) {
    const bool better = split_levels(p, ci, t, s);
    if (threadIdx.x == 0) p.state[ci] = BALANCE;
    if (better) {  // on from there; this pass's sums belong to the old levels
      for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
        p.T[c.vbeg + v] = 0.0;
        p.T2[c.vbeg + v] = 0.0f;
      }
      if (threadIdx.x == 0) {
        lv.since = t + 1;
        lv.split = 1;
        atomicAdd(active, 1u);
      }
      return;
    }
  }
  double *sum = s, *G = s + 32;                     // G: [HIST][HIST + 1]
  double *gamma = G + HIST * (HIST + 1);
  const uint32_t cur = t % (HIST + 1), age = t - lv.since;
  // differences to combine: none once what does not balance has given no order, as the
  // combined steps scatter its weights (463 vertices, all but two of them S: proven in 16
  // of 16 runs, in 5 of 12 with the differences kept; 124 other R-MAT, planted and random
  // graphs at k = 2, 3, 4 take the same time and leave the same four to the flows either way)
  const uint32_t m = age > 18 && !lv.split ? 0 : min(age, (uint32_t)HIST);
  const double total = lv.target[0] * c.n;  // (about the units in all, for relative sizes)
  // (read before block_sum's barriers: thread 0 sets it below, and all threads have to
  // take the same way there)
  const bool wide = __ldcg(p.wide + ci) != 0;
  double over = 0.0;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    const uint32_t g = c.vbeg + v;
    const double wv = __ldcg(p.w + g), T = __ldcg(p.T + g), l = (double)p.k * wv * T;
    over += l > lv.cap ? l - lv.cap : 0.0;
    double slope = 1.0 - (double)__ldcg(p.T2 + g) / (wv * T);  // d log l / d log w
    slope = slope > 1e-3 ? slope : 1e-3;
    p.F[(size_t)cur * p.nv + g] = log(lv.target[p.rest[g]] / l) / slope;
    p.T[g] = 0.0;
    p.T2[g] = 0.0f;
  }
  over = block_sum(over, sum);
  const double rel = over / total;
  // single-precision sums are within about 1e-7: enough while the loads are further
  // apart than that, and for bounds that are far above it
  if (over + (wide ? 0.0 : 2e-7 * total) <= lv.stop) {
    if (threadIdx.x == 0) p.state[ci] = REACHED;
    return;
  }
  if (!wide && rel < 1e-6 && threadIdx.x == 0) p.wide[ci] = 1;
  // not on its way: look for a denser subset, a few times
  if (!(rel < 1e30) || t + 2 >= MAX_PASSES) {
    if (threadIdx.x == 0) p.state[ci] = GIVEN_UP;
    return;
  }
  // (124 solves of R-MAT, planted and random graphs at k = 2, 3, 4: 4 go on to the flows;
  // with orders at ages 5, 9, 13, 17 and 21 9 do, and 24 planted ones take 33.6 ms instead of
  // 30.2; with ages from 12 to 36 4 do and the same take 35.0)
  const bool slow = (age == 8 && rel > 1e-3) || (age == 13 && rel > 1e-4) || (age == 18 && rel > 1e-5) ||
                    age == 23 || age >= 28;
  if (slow && !(lv.split && age == 8)) {
    if (lv.split || lv.orders >= MAX_ORDERS) {  // (S is not the densest, or the rest has levels of its own)
      if (threadIdx.x == 0) p.state[ci] = GIVEN_UP;
      return;
    }
    ask_order(p, ci);
    if (threadIdx.x == 0) {
      lv.orders++;
      p.state[ci] = COUNT;
    }
  }
  if (threadIdx.x == 0) atomicAdd(active, 1u);
  auto F = [&](uint32_t h, uint32_t v) -> double { return p.F[(size_t)(h % (HIST + 1)) * p.nv + c.vbeg + v]; };
  auto X = [&](uint32_t h, uint32_t v) -> double { return p.X[(size_t)(h % (HIST + 1)) * p.nv + c.vbeg + v]; };
  // (over S alone once there is one: the rest, with its own plain steps, need not balance)
  // Gram matrix of the residual differences dF(h) = F(h) - F(h-1) of the last m
  // passes, by slot h mod HIST and kept from one pass to the next, and their products
  // with F(t): of the newest with every other, and of each with F(t), a warp per entry
  double *gram = p.G + (size_t)ci * HIST * HIST;
  for (uint32_t e = threadIdx.x >> 5; e < 2 * m; e += WARPS) {
    const uint32_t r = e >> 1, h = t - r;
    double d = 0.0;
    for (uint32_t v = lane_id(); v < c.n; v += 32) {
      if (p.rest[c.vbeg + v]) continue;
      const double f = F(t, v);
      d += (F(h, v) - F(h - 1, v)) * ((e & 1) ? f : f - F(t - 1, v));
    }
    d = warp_sum(d);
    if (lane_id() == 0) {
      if (e & 1) {
        G[r * (HIST + 1) + m] = d;
      } else {
        gram[h % HIST * HIST + t % HIST] = d;
        gram[t % HIST * HIST + h % HIST] = d;
      }
    }
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < m * m; e += blockDim.x)
    G[e / m * (HIST + 1) + e % m] = gram[(t - e / m) % HIST * HIST + (t - e % m) % HIST];
  __syncthreads();
  if (threadIdx.x < 32) {  // Gauss-Jordan, a column a lane; a trace of regularisation
    const uint32_t col = min(lane_id(), m);
    double g[HIST];
#pragma unroll
    for (int r = 0; r < HIST; r++) {
      g[r] = r < (int)m ? G[r * (HIST + 1) + col] : 0.0;
      if (r == (int)col) g[r] *= 1.0 + 1e-10;
    }
#pragma unroll
    for (int r = 0; r < HIST; r++) {
      if (r >= (int)m) break;
      const double d = __shfl_sync(CDS_FULL, g[r], r);
      g[r] = fabs(d) > 1e-300 ? g[r] / d : 0.0;
#pragma unroll
      for (int x = 0; x < HIST; x++) {
        const double f = __shfl_sync(CDS_FULL, g[x], r);
        if (x != r && x < (int)m) g[x] -= f * g[r];
      }
    }
#pragma unroll
    for (int r = 0; r < HIST; r++)
      if (lane_id() == m && r < (int)m) gamma[r] = g[r];
  }
  __syncthreads();
  double top = -1e300;
  double nx[(MAX_N + THREADS - 1) / THREADS];
  int i = 0;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x, i++) {
    const double x = X(t, v);
    double step = F(t, v);
    for (uint32_t r = 0; r < (p.rest[c.vbeg + v] ? 0 : m); r++)
      step -= gamma[r] * (X(t - r, v) - X(t - r - 1, v) + F(t - r, v) - F(t - r - 1, v));
    step = step > 1.5 ? 1.5 : step < -1.5 ? -1.5 : step == step ? step : 0.0;
    nx[i] = x + step;
    top = nx[i] > top ? nx[i] : top;
  }
  top = block_max(top, sum);
  i = 0;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x, i++) {
    p.X[(size_t)((t + 1) % (HIST + 1)) * p.nv + c.vbeg + v] = nx[i];
    const double d = nx[i] - top;
    p.w[c.vbeg + v] = exp(d < -60.0 ? -60.0 : d);
  }
}

template <int K>
__global__ void __launch_bounds__(THREADS, 1) k_certify(CertParams p) {
  __shared__ double s_up[32 + HIST * (HIST + 1) + HIST];
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long tprev = globaltimer_ns();
  auto phase_end = [&](int i) {
    if (p.phase_ns && leader) {
      const unsigned long long now = globaltimer_ns();
      p.phase_ns[i] += now - tprev;
      tprev = now;
    }
  };
  __shared__ uint32_t s_loaded;  // the component whose rows are in place
  if (threadIdx.x == 0) s_loaded = 0xFFFFFFFFu;
  uint32_t t = 0;
  for (; t < MAX_PASSES; t++) {
    if (leader)  // of the next pass
      for (int i = 0; i < 3; i++) p.ctl[3 * i + (t + 1) % 3] = 0;
    pass_over<K, SUMS>(p, 1u << BALANCE | 1u << COUNT, p.ctl + 3 + t % 3, &s_loaded);
    pass_over<K, FIRSTS>(p, 1u << COUNT, p.ctl + 6 + t % 3, &s_loaded);
    if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
    phase_end(0);
    for (uint32_t ci = blockIdx.x; ci < p.ncomp; ci += gridDim.x) {
      const uint32_t st = __ldcg(p.state + ci);
      if (st == BALANCE || st == COUNT) update(p, ci, t, p.ctl + t % 3, s_up);
    }
    if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
    phase_end(1);
    if (!__ldcg(p.ctl + t % 3)) break;
  }
  if (leader) *p.passes = t + 1;
  pass_over<K, SHARES>(p, 1u << REACHED, p.ctl + 9, &s_loaded);
  phase_end(2);
}

// symmetric rows of every component from the covered pairs of core-local ids
// (bits: row a, column b > a); warp per row and word
__global__ void k_cert_rows(const uint32_t *__restrict__ bits, CoreRows r, uint32_t ncore,
                            const uint32_t *__restrict__ core_vertex, const uint32_t *__restrict__ local,
                            const uint32_t *__restrict__ vcnet, const Comp *__restrict__ comp,
                            uint32_t *__restrict__ rows) {
  each_word(r, ncore, core_vertex, bits, [&](uint32_t i, const CoreBand &bd, uint32_t w, uint32_t m) {
    if (!((m >> lane_id()) & 1u)) return;
    const uint32_t la = local[core_vertex[i]], lb = local[core_vertex[bd.lid + w * 32 + lane_id()]];
    const Comp c = comp[vcnet[la]];
    if (!c.W) return;  // not asked
    const uint32_t a = la - c.vbeg, b = lb - c.vbeg;
    atomicOr(rows + c.row + a * c.W + (b >> 5), 1u << (b & 31));
    atomicOr(rows + c.row + b * c.W + (a >> 5), 1u << (a & 31));
  });
}
// per local vertex: its later neighbours, and the start of the balancing
__device__ __forceinline__ uint32_t later_word(const uint32_t *rows, const Comp &c, uint32_t v, uint32_t x) {
  const uint32_t m = rows[c.row + v * c.W + x];
  return x < (v >> 5) ? 0u : x > (v >> 5) ? m : m & ~((2u << (v & 31)) - 1u);
}
__global__ void k_cert_start(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ vcnet,
                             const Comp *__restrict__ comp, uint32_t nv, uint32_t *__restrict__ cnt,
                             double *__restrict__ w, double *__restrict__ X) {
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < nv; g += gridDim.x * blockDim.x) {
    const Comp c = comp[vcnet[g]];
    uint32_t n = 0;
    for (uint32_t x = 0; x < c.W; x++) n += __popc(later_word(rows, c, g - c.vbeg, x));
    cnt[g] = n;
    w[g] = c.W ? 1.0 : 0.0;  // (not asked)
    X[g] = 0.0;
  }
}
// the edges u < i of every component; its first and their number into comp
__global__ void k_cert_items(const uint32_t *__restrict__ rows, const uint32_t *__restrict__ vcnet,
                             Comp *__restrict__ comp, uint32_t nv, const uint64_t *__restrict__ first,
                             uint32_t *__restrict__ item_u, uint32_t *__restrict__ item_i) {
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < nv; g += warps) {
    const Comp c = comp[vcnet[g]];
    const uint32_t v = g - c.vbeg;
    const uint32_t m = lane_id() < c.W ? later_word(rows, c, v, lane_id()) : 0u;
    uint64_t at = first[g] + warp_inclusive_scan((uint32_t)__popc(m)) - __popc(m);
    for (uint32_t x = m; x; x &= x - 1) {
      item_u[at] = v;
      item_i[at++] = lane_id() * 32 + __ffs(x) - 1;
    }
    if (v == 0 && lane_id() == 0) {
      comp[vcnet[g]].item = (uint32_t)first[g];
      comp[vcnet[g]].nitems = (uint32_t)(first[g + c.n] - first[g]) * c.split;
    }
  }
}

}  // namespace

namespace cds {

void certify(cds_ctx *c, cudaStream_t s, const CoreOut &co, uint32_t k, const std::vector<CertAsk> &ask,
             std::vector<CertAnswer> &out, std::vector<uint8_t> &in_set, DBuf<double> &weights) {
  const uint32_t nnet = co.ncomp, nv = nnet ? co.comp_vbeg[nnet] : 0;
  out.assign(nnet, CertAnswer{});
  in_set.clear();
  if (!co.small || k > 5) return;
  std::vector<Comp> hc(nnet);
  std::vector<uint32_t> hstate(nnet, NOT_ASKED), asked;
  std::vector<Level> hl(nnet);
  uint32_t words = 0;
  uint64_t pairs = 0, work = 0;
  size_t smem = 0;
  for (uint64_t x : co.pruned_edges) pairs += x;
  for (uint32_t i = 0; i < nnet; i++) {
    Comp &h = hc[i];
    h.vbeg = co.comp_vbeg[i];
    h.n = co.comp_vbeg[i + 1] - h.vbeg;
    const uint64_t psi = co.comp_cbeg[i + 1] - co.comp_cbeg[i];
    if (!ask[i].q || h.n > MAX_N || !psi || psi > MAX_CLIQUES) continue;
    h.W = ((h.n + 31) / 32) | 1u;
    if (h.W > 32) h.W = 32;  // a lane a word (1,024 vertices: rows share banks)
    h.row = words;
    words += h.n * h.W;
    const uint32_t per = h.W * ((h.W + ITEM_WORDS - 1) / ITEM_WORDS);
    h.nitems = k == 2 ? per : k == 3 ? h.n * per : 0;
    // small components have few edges: their work is dealt in finer pieces
    h.split = k == 4 && h.n <= 128 ? (h.n + 31) / 32 : k == 5 && h.n <= 256 ? 8 : 1;
    Level &l = hl[i];
    l = Level{};
    l.target[0] = (double)k * (double)psi / (double)h.n;
    l.cap = (double)k * (double)ask[i].p / (double)ask[i].q;
    l.stop = 0.3 * (double)k / (double)ask[i].q;
    l.p = (unsigned long long)ask[i].p;
    l.q = (unsigned long long)ask[i].q;
    hstate[i] = BALANCE;
    asked.push_back(i);
    work += psi;
    smem = std::max(smem, shared_bytes(h.n, h.W));
  }
  if (asked.empty()) return;
  // Parts, shared among the components by their cliques (at most a warp per prefix
  // each): with several, some a block, so that the blocks of a finished component work
  // for the others (19 components of 25 M 4-cliques, two of which never balance:
  // 19.4 -> 6.2 ms).  One component is dealt to the blocks evenly in any case, and a
  // part each spares them the ends of more (988 vertices: 55 -> 42 ms).
  const uint32_t avail = coop_grid(c, 1), per_block = asked.size() > 1 ? PARTS : 1;
  std::vector<Part> parts;
  for (uint32_t i : asked) {
    const uint64_t psi = co.comp_cbeg[i + 1] - co.comp_cbeg[i];
    const uint64_t items = k <= 3 ? hc[i].nitems : std::max<uint64_t>(hc[i].n, psi / 64) * hc[i].split;
    const uint64_t want = (uint64_t)((double)avail * per_block * (double)psi / (double)work) + (asked.size() > 1);
    const uint32_t n = (uint32_t)std::max<uint64_t>(1, std::min(want, (items + WARPS - 1) / WARPS));
    for (uint32_t x = 0; x < n; x++) parts.push_back(Part{i, x, n});
  }
  const unsigned blocks = (unsigned)std::min<size_t>(avail, parts.size());
  DBuf<Comp> comp(c, s, nnet);
  DBuf<Part> d_part(c, s, parts.size());
  DBuf<Level> level(c, s, nnet);
  DBuf<uint32_t> state(c, s, nnet), wide(c, s, nnet), rest(c, s, nv), rank(c, s, nv), firsts(c, s, nv), rows(c, s, words), cnt(c, s, nv), item_u(c, s, k < 4 ? 0 : pairs + 1),
      item_i(c, s, k < 4 ? 0 : pairs + 1), ctl(c, s, 32 + 10 + 2);
  DBuf<uint64_t> first(c, s, nv + 1);
  DBuf<double> w(c, s, nv), T(c, s, nv), X(c, s, (size_t)(HIST + 1) * nv), F(c, s, (size_t)(HIST + 1) * nv),
      G(c, s, (size_t)nnet * HIST * HIST);
  DBuf<float> T2(c, s, nv);
  DBuf<unsigned long long> load(c, s, 2 * (size_t)nv);
  CDS_CUDA(cudaMemcpyAsync(comp.p, hc.data(), nnet * sizeof(Comp), cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(level.p, hl.data(), nnet * sizeof(Level), cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(state.p, hstate.data(), nnet * 4, cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(d_part.p, parts.data(), parts.size() * sizeof(Part), cudaMemcpyHostToDevice, s));
  rows.zero();
  T.zero();
  T2.zero();
  wide.zero();
  rest.zero();
  load.zero();
  ctl.zero();
  const int grid = c->sm_count * 4;
  k_cert_rows<<<grid, 256, 0, s>>>(co.bits.p, co.rows, co.ncore, co.core_vertex.p, co.local.p, co.vcnet.p, comp.p,
                                rows.p);
  k_cert_start<<<(nv + 255) / 256, 256, 0, s>>>(rows.p, co.vcnet.p, comp.p, nv, cnt.p, w.p, X.p);
  count_launch(2);
  if (k > 3) {
    scan_u32(cnt.p, first.p, nv, c, s);
    k_cert_items<<<grid, 256, 0, s>>>(rows.p, co.vcnet.p, comp.p, nv, first.p, item_u.p, item_i.p);
    count_launch();
  }
  CDS_CUDA(cudaGetLastError());
  CertParams p{};
  p.k = k;
  p.ncomp = nnet;
  p.nv = nv;
  p.comp = comp.p;
  p.rows = rows.p;
  p.item_u = item_u.p;
  p.item_i = item_i.p;
  p.part = d_part.p;
  p.nparts = (uint32_t)parts.size();
  p.state = state.p;
  p.wide = wide.p;
  p.level = level.p;
  p.rest = rest.p;
  p.rank = rank.p;
  p.first = firsts.p;
  p.w = w.p;
  p.T = T.p;
  p.T2 = T2.p;
  p.load = load.p;
  p.X = X.p;
  p.F = F.p;
  p.G = G.p;
  static_assert(sizeof(GridBarrier) == 32 * sizeof(uint32_t), "the barrier takes the first line");
  p.bar = reinterpret_cast<GridBarrier *>(ctl.p);
  p.ctl = ctl.p + 32;
  p.err = ctl.p + 42;
  p.passes = p.err + 1;
  p.spin_limit = 1ull << 26;
  DBuf<unsigned long long> phase(c, s, c->prof ? 3 : 0);
  phase.zero();
  p.phase_ns = phase.p;
  void *kern = k == 2 ? (void *)k_certify<2> : k == 3 ? (void *)k_certify<3>
             : k == 4 ? (void *)k_certify<4> : (void *)k_certify<5>;
  cudaFuncAttributes fa;
  CDS_CUDA(cudaFuncGetAttributes(&fa, kern));
  CDS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(c->smem_optin - fa.sharedSizeBytes)));
  void *args[] = {&p};
  {
    ProfScope ps(c, s, "certify");
    CDS_CUDA(cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(THREADS), args, smem, s));
  }
  count_launch();
  CDS_CUDA(cudaGetLastError());
  std::vector<unsigned long long> hload(2 * (size_t)nv);
  std::vector<uint32_t> hrest(nv);
  uint32_t status[2] = {0, 0};
  {
    HostReads r(s);
    r.add(hstate.data(), state.p, nnet);
    r.add(hl.data(), level.p, nnet);
    r.add(hrest.data(), rest.p, nv);
    r.add(hload.data(), load.p, hload.size());
    r.add(status, p.err, 2);
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
    auto &a = c->prof_done["certify_passes"];
    a.first += 1;
    a.second += status[1];
    static const char *pn[3] = {"certify_phase_pass", "certify_phase_update", "certify_phase_integer"};
    for (int i = 0; i < 3; i++) {
      auto &b = c->prof_done[pn[i]];
      b.first += 1;
      b.second += hph[i] / 1e6;
    }
  }
  if (status[0]) fail(CDS_ERR_TIMEOUT, "certify: device iteration budget exhausted");
  const __int128 one = (__int128)1 << UNIT_BITS;
  in_set.assign(nv, 0);
  for (uint32_t i : asked) {
    const Comp &h = hc[i];
    const Level &l = hl[i];
    CertAnswer &o = out[i];
    o.tried = true;
    if (l.size) {  // (a subset that the component cannot have: as if none had been found)
      if (!l.psi || l.psi > co.comp_cbeg[i + 1] - co.comp_cbeg[i] || l.size > h.n) continue;
      o.num = (int64_t)l.psi;
      o.den = l.size;
    }
    if (hstate[i] != REACHED) continue;
    const __int128 psi = (__int128)(co.comp_cbeg[i + 1] - co.comp_cbeg[i]);
    const __int128 cap = (__int128)k * l.p * one;  // times q, as all below
    __int128 sum = 0, over = 0, top = 0, room = (__int128)1 << 120;
    uint32_t size = 0;
    for (uint32_t v = 0; v < h.n; v++) {
      const __int128 x = (__int128)hload[h.vbeg + v] + ((__int128)hload[(size_t)nv + h.vbeg + v] << 32);
      sum += x;
      if (x * l.q > cap) over += x * l.q - cap;
      if (!hrest[h.vbeg + v]) {
        top += x;
        size++;
      } else if (cap - x * l.q < room) {
        room = cap - x * l.q;
      }
    }
    if (sum != psi * k * one) fail(CDS_ERR_CUDA, "certify: loads do not add up to the cliques' units");
    bool good = over < (__int128)k * one;
    // a proper subset: it holds the cliques it was said to, and no other vertex can
    // be in a densest set
    if (l.size) good = good && size == l.size && top >= (__int128)k * one * l.psi && room > over;
    if (!good) continue;
    o.proven = true;
    if (l.size)
      for (uint32_t v = 0; v < h.n; v++) in_set[h.vbeg + v] = !hrest[h.vbeg + v];
  }
  weights = std::move(w);
}

}  // namespace cds
