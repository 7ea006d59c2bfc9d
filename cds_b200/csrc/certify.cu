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
// the R-MAT and planted graphs tried (7 to 36 without the derivative); components
// whose densest set is smaller do not converge, which shows after eight passes, and
// go to the flows.
//
// A pass never stores a clique.  The component's covered pairs are a symmetric
// bitmap of its vertices in shared memory; a warp takes a clique of k-2 vertices
// (none for k = 2, a vertex for k = 3, an edge for k = 4), deals the later common
// neighbours j to its lanes, and lane j walks the bits l of its row inside that
// mask, adding 1 / (sum of weights).  Every clique is so met twice, from j and from
// l, and each lane's sum belongs to its own j: met once, the sums of the last
// members need an atomic or a reduction per prefix, which cost five times the
// arithmetic saved.  Bound by instruction issue, about 20 a visit.  The proof itself
// is in integers: a last pass splits k 2^s units of every clique exactly, and the
// host checks E (and that the loads add up to every clique's units) in 128 bits.
//
// Measured against network build, warm split and push-relabel: 40 vertices and 1,499
// triangles 0.39 -> 0.14 ms, 470 vertices and 25,761 edges 0.69 -> 0.25, 112 and
// 1.18 M 4-cliques 1.5 -> 0.38, 746 and 9.3 M triangles 4.4 -> 1.3, 988 and 1.14 G
// 4-cliques 295 -> 47 (and 62 GB of records and lists that are not built).
#include "device_util.cuh"
#include "stages.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

namespace {

constexpr uint32_t MAX_N = 1024;   // vertices of a component: a word of a row per lane
constexpr int THREADS = 1024, WARPS = THREADS / 32;
constexpr int HIST = 8;            // differences Anderson's method combines
constexpr uint32_t MAX_PASSES = 32;
constexpr uint32_t ITEM_WORDS = 2; // k <= 3: words of l an item walks

struct Comp {
  uint32_t vbeg, n;       // local vertices
  uint32_t W, row;        // words a row (odd: lanes on different rows meet different banks), first word
  uint32_t item, nitems;  // its items (k = 4, 5: edges, from `item` on, ...
  uint32_t split;         // ... each split this many ways)
  double target;          // load every vertex would have at the component's own density
  double cap;             // k alpha
  double stop;            // E below this counts as reached
};
struct Part {             // a block's share of a component's prefixes
  uint32_t comp, part, parts;
};

struct CertParams {
  uint32_t k, ncomp, nv;
  const Comp *comp;
  const uint32_t *rows;       // symmetric bitmap rows
  const uint32_t *item_u;     // k = 4, 5: the edges u < i by component (indexes in it)
  const uint32_t *item_i;
  const uint32_t *part_off;   // [blocks+1] each block's parts
  const Part *part;
  uint32_t *wide;             // [ncomp] sums in double precision from now on
  uint32_t *state;            // [ncomp] 0 balancing, 1 reached, 2 given up or not asked
  double *w;                  // [nv]
  double *T;                  // [nv] sum of 1 / (clique's weights) over the vertex's cliques
  float *T2;                  // [nv] the same of the squares
  unsigned long long *load;   // [2 nv] integer loads: low 32-bit halves, high halves summed
  double *X, *F;              // [(HIST+1) * nv] log-weights and residuals of the last passes
  double *G;                  // [ncomp * HIST * HIST] products of residual differences
  uint32_t *ctl;              // active components, by pass mod 3
  GridBarrier *bar;
  uint32_t *err;
  unsigned long long spin_limit;
  uint32_t *passes;
  unsigned long long *phase_ns;  // [3] block 0's time in passes, updates, the integer pass (profiling; null: off)
};
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
// accumulators (the sum, and in single precision the sum of the squares) and
// returns this lane's sums over its j (every clique twice over the
// calls that cover all j), over words [y0, y1) of mask; of the steps of 32 j every
// split-th from g on.  Two words at a time, a visit from each in flight.  WIDE:
// double precision; else single-precision terms, summed in double per j.
template <bool WIDE>
__device__ __forceinline__ double pair_sums(const Shared &sh, uint32_t y0, uint32_t y1, uint32_t W, uint32_t jmask,
                                            uint32_t mask, uint32_t g, uint32_t split, double base, float &squares) {
  const uint32_t lane = lane_id(), incl = warp_inclusive_scan((uint32_t)__popc(jmask));
  const uint32_t total = __shfl_sync(CDS_FULL, incl, 31);
  double tot = 0.0;
  for (uint32_t q0 = 32 * g; q0 < total; q0 += 32 * split) {
    const uint32_t jq = deal(jmask, incl, min(q0 + lane, total - 1));
    const bool on = q0 + lane < total;
    const uint32_t *row = sh.rows + jq * W;
    const double bj = base + sh.w[jq];
    const float bf = (float)bj;
    double s = 0.0, s2 = 0.0;
    float f = 0.0f, f2 = 0.0f, sq = 0.0f;
    for (uint32_t y = y0; y < y1; y += 2) {
      const uint32_t m0 = __shfl_sync(CDS_FULL, mask, y), m1 = y + 1 < y1 ? __shfl_sync(CDS_FULL, mask, y + 1) : 0u;
      if (!(m0 | m1)) continue;
      // a visit from each word a step (absent ones take slot 0's weights, masked out)
      uint32_t a0 = on ? m0 & row[y] : 0u, a1 = on && m1 ? m1 & row[y + 1] : 0u;
      while (a0 | a1) {
        const bool v0 = a0 != 0, v1 = a1 != 0;
        const uint32_t l0 = v0 ? y * 32 + __ffs(a0) - 1 : 0u, l1 = v1 ? y * 32 + 31 + __ffs(a1) : 0u;
        a0 &= a0 - 1;
        a1 &= a1 - 1;
        const float r0 = v0 ? rcp(bf + sh.wf[l0]) : 0.0f, r1 = v1 ? rcp(bf + sh.wf[l1]) : 0.0f;
        if (WIDE) {
          s += newton(bj + sh.w[l0], r0);  // (0 for an absent one)
          s2 += newton(bj + sh.w[l1], r1);
        } else {
          f += r0;
          f2 += r1;
        }
        sq = fmaf(r0, r0, sq);
        sq = fmaf(r1, r1, sq);
      }
    }
    if (WIDE) s += s2;
    else s = (double)f + (double)f2;
    if (s != 0.0) {
      atomicAdd(sh.acc + jq, s);
      atomicAdd(sh.acc2 + jq, sq);
    }
    tot += s;
    squares += sq;
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
      for (uint32_t m = on ? my & row[y] : 0u; m; m &= m - 1) {
        const uint32_t l = y * 32 + __ffs(m) - 1;
        const double wl = sh.w[l], d = base + (wj + wl), inv = newton(d, rcp((float)d));
        unsigned long long a = (unsigned long long)(units * ((j < l ? wj : wl) * inv));  // the smaller one's
        a = a < all ? a : all;
        unsigned long long b = all - a;  // and the larger one's
        if (NP > 0) {
          const unsigned long long z = (unsigned long long)(units * ((j < l ? wl : wj) * inv));
          b = z < b ? z : b;
        }
        sum += j < l ? a : b;
        if (j < l) rem += all - a - b;
      }
    }
    if (sum) give(j, sum);
  }
  if (NP == 0) return;
  rem = warp_sum(rem);
  if (lane == 0 && rem) {
    unsigned long long left = rem;
#pragma unroll
    for (int x = 1; x < NP; x++) {
      unsigned long long a = (unsigned long long)((double)rem * (sh.w[pre[x]] / base));
      a = a < left ? a : left;
      left -= a;
      give(pre[x], a);
    }
    if (left) give(pre[0], left);
  }
}

// One pass of this block over its parts of the components in state `want`.
template <int K, bool INT>
__device__ __noinline__ void pass_over(const CertParams &p, uint32_t want, bool reload) {
  extern __shared__ __align__(16) char smem[];
  __shared__ uint32_t s_next;  // the next item
  const uint32_t lane = lane_id();
  for (uint32_t x = p.part_off[blockIdx.x]; x < p.part_off[blockIdx.x + 1]; x++) {
    const Part pt = p.part[x];
    if (__ldcg(p.state + pt.comp) != want) continue;
    const Comp c = p.comp[pt.comp];
    __syncthreads();
    Shared sh;
    sh.w = reinterpret_cast<double *>(smem);
    sh.acc = sh.w + c.n;
    sh.wf = reinterpret_cast<float *>(sh.acc + c.n);
    sh.acc2 = sh.wf + c.n;
    sh.rows = reinterpret_cast<uint32_t *>(sh.acc2 + c.n);
    if (reload || p.part_off[blockIdx.x + 1] - p.part_off[blockIdx.x] > 1) {  // else in place from the first pass
      for (uint32_t i = threadIdx.x; i < c.n * c.W; i += blockDim.x) sh.rows[i] = p.rows[c.row + i];
    }
    for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
      const double w = __ldcg(p.w + c.vbeg + v);
      sh.w[v] = w;
      sh.wf[v] = (float)w;
      sh.acc[v] = 0.0;
      sh.acc2[v] = 0.0f;
    }
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
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
      if constexpr (INT) {
        pair_shares<K - 2>(sh, y0, y1, c.W, jmask, mask, g, split, base, p.k, pre, lo, hi);
      } else {
        float sq = 0.0f;
        const double t = wide ? pair_sums<true>(sh, y0, y1, c.W, jmask, mask, g, split, base, sq)
                              : pair_sums<false>(sh, y0, y1, c.W, jmask, mask, g, split, base, sq);
        if constexpr (K > 2) {
          const double h = 0.5 * warp_sum(t);
          sq = 0.5f * warp_sum(sq);
          if (lane < K - 2) {
            atomicAdd(sh.acc + pre[lane < K - 2 ? lane : 0], h);
            atomicAdd(sh.acc2 + pre[lane < K - 2 ? lane : 0], sq);
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
    __syncthreads();
    if (!INT)
      for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x)
        if (sh.acc[v] != 0.0) {
          atomicAdd(p.T + c.vbeg + v, sh.acc[v]);
          atomicAdd(p.T2 + c.vbeg + v, sh.acc2[v]);
        }
  }
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

// After pass t: the loads of component ci, and its next weights.  One block; the
// same block takes the component every time, so its history is its own.
__device__ __noinline__ void update(const CertParams &p, uint32_t ci, uint32_t t, uint32_t *active, double *s) {
  const Comp c = p.comp[ci];
  double *sum = s, *G = s + 32;                     // G: [HIST][HIST + 1]
  double *gamma = G + HIST * (HIST + 1);
  const uint32_t cur = t % (HIST + 1), m = min(t, (uint32_t)HIST);
  double over = 0.0;
  for (uint32_t v = threadIdx.x; v < c.n; v += blockDim.x) {
    const uint32_t g = c.vbeg + v;
    const double wv = __ldcg(p.w + g), T = __ldcg(p.T + g), l = (double)p.k * wv * T;
    over += l > c.cap ? l - c.cap : 0.0;
    double slope = 1.0 - wv * (double)__ldcg(p.T2 + g) / T;  // d log l / d log w
    slope = slope > 1e-3 ? slope : 1e-3;
    p.F[(size_t)cur * p.nv + g] = log(c.target / l) / slope;
    p.T[g] = 0.0;
    p.T2[g] = 0.0f;
  }
  over = block_sum(over, sum);
  const double rel = over / (c.target * c.n);
  // single-precision sums are within about 1e-7: enough while the loads are further
  // apart than that, and for bounds that are far above it
  const bool wide = __ldcg(p.wide + ci) != 0;
  if (over + (wide ? 0.0 : 2e-7 * c.target * c.n) <= c.stop) {
    if (threadIdx.x == 0) p.state[ci] = 1;
    return;
  }
  if (!wide && rel < 1e-6 && threadIdx.x == 0) p.wide[ci] = 1;
  // not on its way: a component that some subset of it is denser than
  if (!(rel < 1e30) || (t >= 8 && rel > 1e-3) || (t >= 12 && rel > 1e-4) || (t >= 16 && rel > 1e-5) ||
      (t >= 20 && rel > 1e-6) || t + 1 >= MAX_PASSES) {
    if (threadIdx.x == 0) p.state[ci] = 2;
    return;
  }
  if (threadIdx.x == 0) atomicAdd(active, 1u);
  auto F = [&](uint32_t h, uint32_t v) -> double { return p.F[(size_t)(h % (HIST + 1)) * p.nv + c.vbeg + v]; };
  auto X = [&](uint32_t h, uint32_t v) -> double { return p.X[(size_t)(h % (HIST + 1)) * p.nv + c.vbeg + v]; };
  // Gram matrix of the residual differences dF(h) = F(h) - F(h-1) of the last m
  // passes, by slot h mod HIST and kept from one pass to the next, and their products
  // with F(t): of the newest with every other, and of each with F(t), a warp per entry
  double *gram = p.G + (size_t)ci * HIST * HIST;
  for (uint32_t e = threadIdx.x >> 5; e < 2 * m; e += WARPS) {
    const uint32_t r = e >> 1, h = t - r;
    double d = 0.0;
    for (uint32_t v = lane_id(); v < c.n; v += 32) {
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
    for (uint32_t r = 0; r < m; r++)
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
  uint32_t t = 0;
  for (; t < MAX_PASSES; t++) {
    if (leader) p.ctl[(t + 1) % 3] = 0;  // of the next pass
    pass_over<K, false>(p, 0, t == 0);
    if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
    phase_end(0);
    for (uint32_t ci = blockIdx.x; ci < p.ncomp; ci += gridDim.x)
      if (__ldcg(p.state + ci) == 0) update(p, ci, t, p.ctl + t % 3, s_up);
    if (!grid_sync(p.bar, p.err, p.spin_limit)) return;
    phase_end(1);
    if (!__ldcg(p.ctl + t % 3)) break;
  }
  if (leader) *p.passes = t + 1;
  pass_over<K, true>(p, 1, false);
  phase_end(2);
}

// symmetric rows of every component from the covered pairs of core-local ids
// (bits: row a, column b > a); warp per row and word
__global__ void k_cert_rows(const uint32_t *__restrict__ bits, uint32_t words, uint32_t ncore,
                            const uint32_t *__restrict__ core_vertex, const uint32_t *__restrict__ local,
                            const uint32_t *__restrict__ vcnet, const Comp *__restrict__ comp,
                            uint32_t *__restrict__ rows) {
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5, total = ncore * words;
  for (uint32_t x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < total; x += warps) {
    const uint32_t m = bits[x];
    if (!((m >> lane_id()) & 1u)) continue;
    const uint32_t la = local[core_vertex[x / words]], lb = local[core_vertex[x % words * 32 + lane_id()]];
    const Comp c = comp[vcnet[la]];
    if (!c.W) continue;  // not asked
    const uint32_t a = la - c.vbeg, b = lb - c.vbeg;
    atomicOr(rows + c.row + a * c.W + (b >> 5), 1u << (b & 31));
    atomicOr(rows + c.row + b * c.W + (a >> 5), 1u << (a & 31));
  }
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
             std::vector<uint8_t> &proven, DBuf<double> &weights) {
  const uint32_t nnet = co.ncomp, nv = nnet ? co.comp_vbeg[nnet] : 0;
  proven.assign(nnet, 0);
  if (!co.small || k > 5) return;
  std::vector<Comp> hc(nnet);
  std::vector<uint32_t> hstate(nnet, 2), asked;
  uint32_t words = 0;
  uint64_t pairs = 0, work = 0;
  size_t smem = 0;
  for (uint64_t x : co.pruned_edges) pairs += x;
  for (uint32_t i = 0; i < nnet; i++) {
    Comp &h = hc[i];
    h.vbeg = co.comp_vbeg[i];
    h.n = co.comp_vbeg[i + 1] - h.vbeg;
    const uint64_t psi = co.comp_cbeg[i + 1] - co.comp_cbeg[i];
    if (!ask[i].q || h.n > MAX_N || !psi) continue;
    h.W = ((h.n + 31) / 32) | 1u;
    if (h.W > 32) h.W = 32;  // a lane a word (1,024 vertices: rows share banks)
    h.row = words;
    words += h.n * h.W;
    const uint32_t per = h.W * ((h.W + ITEM_WORDS - 1) / ITEM_WORDS);
    h.nitems = k == 2 ? per : k == 3 ? h.n * per : 0;
    // small components have few edges: their work is dealt in finer pieces
    h.split = k == 4 && h.n <= 128 ? (h.n + 31) / 32 : k == 5 && h.n <= 256 ? 8 : 1;
    h.target = (double)k * (double)psi / (double)h.n;
    h.cap = (double)k * (double)ask[i].p / (double)ask[i].q;
    h.stop = 0.3 * (double)k / (double)ask[i].q;
    hstate[i] = 0;
    asked.push_back(i);
    work += psi;
    smem = std::max(smem, shared_bytes(h.n, h.W));
  }
  if (asked.empty()) return;
  // Blocks: one an SM at most.  Every component gets its share of them by cliques
  // (at least one, at most a warp per prefix); with more components than blocks,
  // the largest go first to the block with the least work.
  const uint32_t avail = coop_grid(c, 1);
  std::vector<std::vector<Part>> plan;
  if (asked.size() <= avail) {
    for (uint32_t i : asked) {
      const uint64_t psi = co.comp_cbeg[i + 1] - co.comp_cbeg[i];
      const uint64_t prefixes = k <= 3 ? hc[i].nitems : std::max<uint64_t>(hc[i].n, psi / 64);
      uint64_t parts = (avail - asked.size()) * psi / work + 1;
      parts = std::max<uint64_t>(1, std::min(parts, (prefixes + WARPS - 1) / WARPS));
      for (uint32_t x = 0; x < parts; x++) plan.push_back({Part{i, x, (uint32_t)parts}});
    }
  } else {
    std::vector<uint32_t> order = asked;
    std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
      const uint64_t x = co.comp_cbeg[a + 1] - co.comp_cbeg[a], y = co.comp_cbeg[b + 1] - co.comp_cbeg[b];
      return x != y ? x > y : a < b;
    });
    plan.resize(avail);
    std::vector<uint64_t> sum(avail, 0);
    for (uint32_t i : order) {
      const size_t b = (size_t)(std::min_element(sum.begin(), sum.end()) - sum.begin());
      plan[b].push_back(Part{i, 0, 1});
      sum[b] += co.comp_cbeg[i + 1] - co.comp_cbeg[i];
    }
  }
  std::vector<uint32_t> off(plan.size() + 1, 0);
  std::vector<Part> parts;
  for (size_t b = 0; b < plan.size(); b++) {
    parts.insert(parts.end(), plan[b].begin(), plan[b].end());
    off[b + 1] = (uint32_t)parts.size();
  }
  DBuf<Comp> comp(c, s, nnet);
  DBuf<Part> d_part(c, s, parts.size());
  DBuf<uint32_t> state(c, s, nnet), wide(c, s, nnet), rows(c, s, words), cnt(c, s, nv), item_u(c, s, k < 4 ? 0 : pairs + 1),
      item_i(c, s, k < 4 ? 0 : pairs + 1), ctl(c, s, 32 + 3 + 2), d_off(c, s, off.size());
  DBuf<uint64_t> first(c, s, nv + 1);
  DBuf<double> w(c, s, nv), T(c, s, nv), X(c, s, (size_t)(HIST + 1) * nv), F(c, s, (size_t)(HIST + 1) * nv),
      G(c, s, (size_t)nnet * HIST * HIST);
  DBuf<float> T2(c, s, nv);
  DBuf<unsigned long long> load(c, s, 2 * (size_t)nv);
  CDS_CUDA(cudaMemcpyAsync(comp.p, hc.data(), nnet * sizeof(Comp), cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(state.p, hstate.data(), nnet * 4, cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(d_off.p, off.data(), off.size() * 4, cudaMemcpyHostToDevice, s));
  CDS_CUDA(cudaMemcpyAsync(d_part.p, parts.data(), parts.size() * sizeof(Part), cudaMemcpyHostToDevice, s));
  rows.zero();
  T.zero();
  T2.zero();
  wide.zero();
  load.zero();
  ctl.zero();
  const int grid = c->sm_count * 4;
  k_cert_rows<<<grid, 256, 0, s>>>(co.bits.p, co.words, co.ncore, co.core_vertex.p, co.local.p, co.vcnet.p, comp.p,
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
  p.part_off = d_off.p;
  p.part = d_part.p;
  p.state = state.p;
  p.wide = wide.p;
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
  p.err = ctl.p + 35;
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
    CDS_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)plan.size()), dim3(THREADS), args, smem, s));
  }
  count_launch();
  CDS_CUDA(cudaGetLastError());
  std::vector<unsigned long long> hload(2 * (size_t)nv);
  uint32_t status[2] = {0, 0};
  {
    HostReads r(s);
    r.add(hstate.data(), state.p, nnet);
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
  for (uint32_t i : asked) {
    if (hstate[i] != 1) continue;
    const Comp &h = hc[i];
    const __int128 psi = (__int128)(co.comp_cbeg[i + 1] - co.comp_cbeg[i]);
    const __int128 cap = (__int128)k * ask[i].p * one;  // times q
    __int128 sum = 0, over = 0;
    for (uint32_t v = 0; v < h.n; v++) {
      const __int128 l = (__int128)hload[h.vbeg + v] + ((__int128)hload[(size_t)nv + h.vbeg + v] << 32);
      sum += l;
      if (l * ask[i].q > cap) over += l * ask[i].q - cap;
    }
    if (sum != psi * k * one) fail(CDS_ERR_CUDA, "certify: loads do not add up to the cliques' units");
    proven[i] = over < (__int128)k * one;
  }
  weights = std::move(w);
}

}  // namespace cds
