// guide_tree.cu -- UPGMA / neighbour-joining guide trees from all-vs-all
// identities, on the GPU.
//
// This is the step the external multiple aligners run after their
// all-vs-all stage (the editor asks ClustalO for tree order,
// tweakseq/Core/ClustalO.cpp:51); the reference itself has no tree code, so
// the definition is the published methods (UPGMA: Sokal & Michener 1958;
// neighbour joining: Saitou & Nei 1987 in the Studier & Keppler 1988 form)
// over integer fixed-point distances (units of 2^-32).  Integers make every
// step exact: the result does not depend on summation order, and GB300's
// integer pipes are full rate where FP64 is not.
//
// Layout.  D is an n x n int64 matrix (row stride n) over *slots*: the m
// active clusters always occupy slots 0..m-1.  A join keeps the cluster at
// slot i and moves the last slot into slot j, so every scan reads a dense
// m x m upper triangle.  Each slot carries its canonical position (the
// position the textbook algorithm would give it: join t takes the smaller
// position of its children), so ties break exactly as in the position-
// ordered definition: smallest criterion, then smallest position pair.
//
// Up to kClusterLeaves active clusters, all joins run in one launch of one
// thread-block cluster (tree_cluster_kernel).  Above that, two launches per
// join.  The scan: every block scans a share of the triangle (rows folded in
// pairs a, m-2-a so each share has m entries) and writes its best candidate;
// the last block to finish (atomic ticket, no waiting) picks and records the
// join.  The join: one thread per remaining slot updates the joined cluster's
// distances, the NJ row sums and the move of the last slot into the freed one.
// The host issues these launches with grids sized for the active count m =
// n - t, which it knows.
#include <climits>
#include <cstring>
#include <map>
#include <mutex>

#include <cooperative_groups.h>

#include "engine.h"

namespace tsq {
namespace {

constexpr int kTreeThreads = 256;

struct TreeState {
  int32_t m, t;
  uint32_t ticket;
  int32_t error;
  // The join the scan picked, for the join launch: slots i and j (pos[i] is
  // the smaller canonical position lo), the slot a the joined cluster takes
  // (i unless i is the last slot), the slot f that frees up, and the last
  // slot L that moves into f.
  int32_t i, j, a, f, L, lo, si, sj;
  int64_t dij;
};

struct Cand {
  int64_t c;
  int32_t lo, hi;  // canonical positions, lo < hi
  int32_t sa, sb;  // slots
};

__device__ __forceinline__ bool better(const Cand &x, const Cand &y) {
  if (x.c != y.c) return x.c < y.c;
  if (x.lo != y.lo) return x.lo < y.lo;
  return x.hi < y.hi;
}

__device__ __forceinline__ Cand shfl_cand(const Cand &x, int src) {
  Cand y;
  y.c = __shfl_sync(0xffffffffu, x.c, src);
  y.lo = __shfl_sync(0xffffffffu, x.lo, src);
  y.hi = __shfl_sync(0xffffffffu, x.hi, src);
  y.sa = __shfl_sync(0xffffffffu, x.sa, src);
  y.sb = __shfl_sync(0xffffffffu, x.sb, src);
  return y;
}

__device__ Cand block_best(Cand x, Cand *sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const Cand y = shfl_cand(x, (lane + o) & 31);
    if (better(y, x)) x = y;
  }
  if (lane == 0) sm[w] = x;
  __syncthreads();
  if (w == 0) {
    x = lane < kTreeThreads / 32 ? sm[lane] : sm[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const Cand y = shfl_cand(x, (lane + o) & 31);
      if (better(y, x)) x = y;
    }
    if (lane == 0) sm[0] = x;
  }
  __syncthreads();
  const Cand r = sm[0];
  __syncthreads();
  return r;
}

__device__ int64_t block_sum(int64_t v, int64_t *sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sm[w] = v;
  __syncthreads();
  int64_t s = 0;
  for (int k = 0; k < kTreeThreads / 32; ++k) s += sm[k];
  __syncthreads();
  return s;
}

__device__ __forceinline__ int64_t floor_div(int64_t a, int64_t b) {
  int64_t q = a / b;
  if ((a % b != 0) && ((a < 0) != (b < 0))) --q;
  return q;
}

// floor(v / d) for 0 < d < 2^32, with inv = floor((2^64 - 1) / d): one
// high multiply and at most two corrections.
__device__ __forceinline__ int64_t floor_div_by(int64_t v, uint32_t d, uint64_t inv) {
  const uint64_t x = v < 0 ? ~uint64_t(v) : uint64_t(v);  // (floor of a negative: ~(~v / d))
  uint64_t q = __umul64hi(x, inv);
  uint64_t rem = x - q * d;
  if (rem >= d) {
    ++q;
    rem -= d;
  }
  if (rem >= d) ++q;
  return int64_t(v < 0 ? ~q : q);
}

struct TreeArgs {
  int64_t *D;
  int64_t *r, *height;
  int32_t *pos, *node, *size;
  TreeState *st;
  Cand *partial;
  tsq_tree_node *out;
  int32_t n;
};

// Scan and pick: every block scans its share of the active triangle; the
// last block to finish (atomic ticket, no waiting) picks the join, records
// it and leaves the slots to the join launch.
template <bool NJ>
__global__ void __launch_bounds__(kTreeThreads) tree_scan_kernel(TreeArgs A, int32_t m, int32_t t) {
  __shared__ Cand sm_c[kTreeThreads / 32];
  __shared__ bool last;
  const int32_t n = A.n;
  if (m < 2 || A.st->error) return;
  const int64_t m2 = m - 2;

  Cand best{LLONG_MAX, INT_MAX, INT_MAX, -1, -1};
  const int32_t nfold = m / 2;
  for (int32_t fa = blockIdx.x; fa < nfold; fa += gridDim.x) {
    const int32_t a1 = fa, a2 = m - 2 - fa;
    const int32_t len1 = m - 1 - a1;
    const int32_t len2 = a2 != a1 ? m - 1 - a2 : 0;
    const int64_t r1 = NJ ? A.r[a1] : 0, r2 = NJ ? A.r[a2] : 0;
    const int32_t p1 = A.pos[a1], p2 = A.pos[a2];
    for (int32_t e = threadIdx.x; e < len1 + len2; e += kTreeThreads) {
      const bool first_row = e < len1;
      const int32_t row = first_row ? a1 : a2;
      const int32_t col = first_row ? a1 + 1 + e : a2 + 1 + (e - len1);
      const int64_t d = A.D[int64_t(row) * n + col];
      const int64_t c = NJ ? m2 * d - (first_row ? r1 : r2) - A.r[col] : d;
      if (c > best.c) continue;  // positions are only read for candidates that can win
      const int32_t pr = first_row ? p1 : p2, pc = A.pos[col];
      const Cand x{c, min(pr, pc), max(pr, pc), row, col};
      if (better(x, best)) best = x;
    }
  }
  best = block_best(best, sm_c);
  if (threadIdx.x == 0) {
    A.partial[blockIdx.x] = best;
    __threadfence();
    last = atomicAdd(&A.st->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();

  best = Cand{LLONG_MAX, INT_MAX, INT_MAX, -1, -1};
  for (int k = threadIdx.x; k < int(gridDim.x); k += kTreeThreads) {
    const volatile Cand *vp = A.partial + k;
    const Cand x{vp->c, vp->lo, vp->hi, vp->sa, vp->sb};
    if (better(x, best)) best = x;
  }
  best = block_best(best, sm_c);
  if (threadIdx.x != 0) return;
  A.st->ticket = 0u;
  if (best.sa < 0) {
    A.st->error = 1;  // stops the remaining launches
    return;
  }
  const int32_t i = A.pos[best.sa] == best.lo ? best.sa : best.sb;
  const int32_t j = i == best.sa ? best.sb : best.sa;
  const int64_t dij = A.D[int64_t(i) * n + j];
  const int32_t si = A.size[i], sj = A.size[j];
  tsq_tree_node o;
  o.left = A.node[i];
  o.right = A.node[j];
  o.size = si + sj;
  o.pos = best.lo;
  o.dist = dij;
  if (NJ) {
    o.height = 0;
    o.left_length = m > 2 ? floor_div(m2 * dij + A.r[i] - A.r[j], 2 * m2) : (dij >> 1);
    o.right_length = dij - o.left_length;
  } else {
    const int64_t h = dij >> 1;
    o.height = h;
    o.left_length = h - A.height[i];
    o.right_length = h - A.height[j];
  }
  A.out[t] = o;
  const int32_t L = m - 1;
  const int32_t a = i != L ? i : j;
  A.st->i = i;
  A.st->j = j;
  A.st->a = a;
  A.st->f = a == i ? j : i;
  A.st->L = L;
  A.st->lo = best.lo;
  A.st->si = si;
  A.st->sj = sj;
  A.st->dij = dij;
  A.st->m = m - 1;  // for the host's final check only: the launches take m and t as arguments
  A.st->t = t + 1;
  if (NJ) A.r[a] = 0;  // the join launch adds the new row sum into it
}

// The join: one thread per remaining slot k.  Thread k writes the joined
// cluster's distance to k (row and column a) and, when the last slot L moves
// into the freed slot f, L's distance to k (row and column f); slot L's own
// thread writes the distance between the joined cluster and L at (a, f).
// Every thread touches only its own k's entries of rows/columns a and f and
// reads only rows i, j and L, so the updates are independent.
template <bool NJ>
__global__ void __launch_bounds__(kTreeThreads) tree_join_kernel(TreeArgs A, int32_t m, int32_t t) {
  __shared__ int64_t sm_s[kTreeThreads / 32];
  const TreeState st = *A.st;
  const int32_t n = A.n;
  if (m < 2 || st.error) return;
  const int32_t i = st.i, j = st.j, a = st.a, f = st.f, L = st.L;
  const int64_t dij = st.dij, si = st.si, sj = st.sj;
  const bool move = f != L;
  int64_t rsum = 0;
  for (int32_t k = blockIdx.x * kTreeThreads + threadIdx.x; k < m; k += gridDim.x * kTreeThreads) {
    if (k == i || k == j) continue;
    const int64_t dik = A.D[int64_t(i) * n + k], djk = A.D[int64_t(j) * n + k];
    const int64_t du = NJ ? (dik + djk - dij) >> 1 : floor_div(si * dik + sj * djk, si + sj);
    rsum += du;
    const int64_t rk = NJ ? A.r[k] + du - dik - djk : 0;
    if (move && k == L) {
      // L takes slot f.
      A.D[int64_t(a) * n + f] = du;
      A.D[int64_t(f) * n + a] = du;
      A.D[int64_t(f) * n + f] = 0;
      if (NJ) A.r[f] = rk;
      A.height[f] = A.height[L];
      A.pos[f] = A.pos[L];
      A.node[f] = A.node[L];
      A.size[f] = A.size[L];
    } else {
      A.D[int64_t(a) * n + k] = du;
      A.D[int64_t(k) * n + a] = du;
      if (NJ) A.r[k] = rk;
      if (move) {
        const int64_t dlk = A.D[int64_t(L) * n + k];
        A.D[int64_t(f) * n + k] = dlk;
        A.D[int64_t(k) * n + f] = dlk;
      }
    }
  }
  if (NJ) {
    rsum = block_sum(rsum, sm_s);
    if (threadIdx.x == 0 && rsum != 0) atomicAdd(reinterpret_cast<unsigned long long *>(A.r + a),
                                                 static_cast<unsigned long long>(rsum));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (!NJ) A.height[a] = dij >> 1;
    A.node[a] = n + t;
    A.size[a] = int32_t(si + sj);
    A.pos[a] = st.lo;
    A.D[int64_t(a) * n + a] = 0;
  }
}

// ---- all joins in one cluster ------------------------------------------------
// A join of a few thousand clusters is short work behind a long chain of
// latencies: two launches per join took 15 us whatever m (7.5 us each).  Here
// the CTAs of one cluster keep the slot tables in their own shared memory, each
// a full copy, and meet at hardware cluster barriers: 4.4 us a join at 500
// leaves and 7.3 at 2,003 (NJ), of which about half are the three trips to L2
// and the two barriers.  (Whole calls, before and now: 2,003 leaves NJ 31.2 and
// 14.6 ms; 4,000 leaves, whose first 700 joins take two launches each, UPGMA 91 and
// 56 to 59 ms, NJ 94 and 77 ms; 8 CTAs for 16: 2,003 leaves NJ 20.8 for 16.2 ms;
// 512 threads for 256: 500 leaves 2.99 for 2.66 ms.)
//
// Rows, not the triangle.  Each slot keeps a lower bound of the criterion over
// its whole row and a neighbour whose criterion is known exactly.  The smallest
// of the known ones, ub, is at least the best criterion, so only rows whose
// bound is at most ub can hold the join (or a tie of it); they are scanned
// whole and their bounds become exact.  A join deletes two neighbours (a bound
// stays one) and adds the joined cluster, whose criterion with every row is
// computed.  UPGMA's criterion does not change otherwise: a row whose known
// neighbour attains its bound is settled until that neighbour is joined, and
// only the other rows are scanned (0.7 a join).  NJ's does: with
// delta_k = D(i,k) + D(j,k) - D(u,k), what row sum k loses, q(k,l) changes by
// delta_k + delta_l - D(k,l) >= delta_k + min delta - max D, and the bound moves
// by that.  (Rows scanned per join of 800 leaves: 36 on family identities, 171 on
// unrelated sequences; the triangle is 400.)
//
// Per join:
// 1. every CTA lists the rows whose bound is at most ub (the same list), the
//    cluster's warps share them, a row cut into parts while warps are left;
//    each part's best goes to every CTA's shared memory; barrier A;
// 2. every CTA picks the same join from them, reads the two joined rows and
//    updates its copy of the tables; barrier B (arrived at once the rows are
//    read) separates these reads from step 3;
// 3. each CTA writes its share of the new distances: row and column a (the
//    joined cluster) and f (the last slot L, moved).
// The next scan does not wait for step 3: it takes column and row a from du, f
// from column and row L, and passes over columns a and f as stored, whose
// values may be on their way.  Barrier A of the next join makes the writes
// visible to step 2.  Distances are read past L1 (other CTAs write them).
constexpr int kClusterThreads = 256, kClusterWarps = kClusterThreads / 32;
constexpr int kMaxClusterCtas = 16;
constexpr int kRefresh = 1024;  // results per join that are kept (row parts)
// Bytes per slot: r, du, bound, near_d (8 each), pos, node, size, near, list.
constexpr int kSlotBytes = 52;
constexpr int kClusterLeaves = 3300;  // what the tables leave room for in 227 KB
constexpr int kMaskWords = (kClusterLeaves + 31) / 32;
// A bound below every criterion, with room for the drift of all joins.
constexpr int64_t kUnknown = LLONG_MIN / 2;

struct WideCand {
  int64_t c, d;  // criterion, distance
  int32_t lo, hi, sa, sb;
};

// Whether criterion c at positions lo, hi comes before x.
__device__ __forceinline__ bool better_pair(const WideCand &x, int64_t c, int32_t lo, int32_t hi) {
  return c < x.c || (c == x.c && (lo < x.lo || (lo == x.lo && hi < x.hi)));
}

// What a row part's scan found: the least criterion, its distance and slot.
struct Refresh {
  int64_t c, d;
  int32_t row, near;
};

// 64-bit warp reductions from the 32-bit redux instructions (a shuffle tree
// takes ten shuffles and twice the time).
__device__ __forceinline__ int64_t warp_min(int64_t v) {
  const int32_t hi = int32_t(v >> 32), bh = __reduce_min_sync(0xffffffffu, hi);
  const uint32_t bl = __reduce_min_sync(0xffffffffu, hi == bh ? uint32_t(v) : 0xffffffffu);
  return int64_t((uint64_t(uint32_t(bh)) << 32) | bl);
}
__device__ __forceinline__ int64_t warp_max(int64_t v) { return ~warp_min(~v); }
__device__ __forceinline__ int64_t warp_sum(int64_t v) {  // (modulo 2^64, by 16-bit pieces)
  uint64_t s = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    s += uint64_t(__reduce_add_sync(0xffffffffu, uint32_t(uint64_t(v) >> (16 * q)) & 0xFFFFu)) << (16 * q);
  return int64_t(s);
}

// The lane holding the smallest (c, lo, hi) of the warp.
__device__ __forceinline__ int best_lane(int64_t c, int32_t lo, int32_t hi) {
  unsigned who = __ballot_sync(0xffffffffu, c == warp_min(c));
  if (__popc(who) > 1) {
    const bool in = (who >> (threadIdx.x & 31)) & 1u;
    const int32_t bl = __reduce_min_sync(0xffffffffu, in ? lo : INT_MAX);
    const int32_t bh = __reduce_min_sync(0xffffffffu, in && lo == bl ? hi : INT_MAX);
    who = __ballot_sync(0xffffffffu, in && lo == bl && hi == bh);
  }
  return __ffs(who) - 1;
}

template <bool NJ>
__global__ void __launch_bounds__(kClusterThreads, 1) tree_cluster_kernel(TreeArgs A, int32_t m0, int32_t t0) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint8_t tree_smem[];
  __shared__ WideCand s_warp[kClusterWarps], s_joined[kClusterWarps];
  __shared__ WideCand s_cand[kMaxClusterCtas];
  __shared__ int64_t s_red[4][kMaxClusterCtas];  // (kClusterWarps entries as well)
  __shared__ uint32_t s_mask[kMaskWords];
  static_assert(kMaskWords <= 128, "four words per lane");
  static_assert(kClusterWarps <= kMaxClusterCtas && kClusterWarps <= 32, "reduction slots");
  Refresh *refresh = reinterpret_cast<Refresh *>(tree_smem);
  int64_t *r = reinterpret_cast<int64_t *>(refresh + kRefresh);
  int64_t *du = r + m0, *bound = du + m0, *near_d = bound + m0;
  int32_t *pos = reinterpret_cast<int32_t *>(near_d + m0), *node = pos + m0, *size = node + m0, *near = size + m0;
  int32_t *list = near + m0;
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t n = A.n;
  if (A.st->error) return;  // (the same for every CTA)
  for (int k = tid; k < m0; k += kClusterThreads) {
    r[k] = A.r[k];
    pos[k] = A.pos[k];
    node[k] = A.node[k];
    size[k] = A.size[k];
    bound[k] = kUnknown;  // every row is scanned for the first join
    near[k] = -1;
  }
  __syncthreads();
  // Minimum over the CTA's threads (NJ: sum and maximum as well), for every
  // thread; one barrier.  Two uses of one slot have another barrier between.
  auto block_min = [&](int64_t v, int slot) {
    v = warp_min(v);
    if (lane == 0) s_red[slot][warp] = v;
    __syncthreads();
    return warp_min(s_red[slot][lane % kClusterWarps]);
  };
  auto block_sum_min_max = [&](int64_t &sum, int64_t &mn, int64_t &mx) {
    sum = warp_sum(sum);
    mx = warp_max(mx);
    if (lane == 0) {
      s_red[0][warp] = sum;
      s_red[1][warp] = mx;
    }
    mn = block_min(mn, 2);
    sum = warp_sum(lane < kClusterWarps ? s_red[0][lane] : 0);
    mx = warp_max(s_red[1][lane % kClusterWarps]);
  };
  int64_t dmax = LLONG_MIN;  // NJ: at least every distance between active slots
  if (NJ) {
    for (int row = rank * kClusterWarps + warp; row < m0; row += ctas * kClusterWarps) {
      const int64_t *p = A.D + row * n;
#pragma unroll 8
      for (int col = lane; col < m0; col += 32) {
        const int64_t d = __ldcg(p + col);
        if (col != row && d > dmax) dmax = d;
      }
    }
    int64_t sum = 0, mn = 0;
    block_sum_min_max(sum, mn, dmax);
    cluster.sync();  // (every CTA has read its s_red)
    if (warp == 0 && lane < ctas) *cluster.map_shared_rank(&s_red[0][rank], lane) = dmax;
    cluster.sync();
    for (int c = 0; c < ctas; ++c) dmax = s_red[0][c] > dmax ? s_red[0][c] : dmax;
    cluster.sync();
  }

  int64_t ub = LLONG_MAX;
  WideCand settled{LLONG_MAX, 0, INT_MAX, INT_MAX, -1, -1};  // UPGMA: the best pair of the settled rows
  int a = -1, f = m0, src_f = 0;  // the last join's slots (f = m: no slot moved); row f is still at row src_f
  for (int m = m0, t = t0; m >= 2; --m, ++t) {
    const int64_t m2 = m - 2;
    // ---- 1. list and scan rows ----
    const int words = (m + 31) >> 5;
    for (int w = warp; w < words; w += kClusterWarps) {
      const int k = 32 * w + lane;
      const int kk = k < m ? k : 0;
      const bool open = NJ || near[kk] < 0 || near_d[kk] != bound[kk];
      const unsigned b = __ballot_sync(0xffffffffu, k < m && open && bound[kk] <= ub);
      if (lane == 0) s_mask[w] = b;
    }
    __syncthreads();
    int rows;
    {
      // Set bits before each word: lane q holds words 4q .. 4q + 3.
      int c[4], incl = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c[q] = incl;
        incl += 4 * lane + q < words ? __popc(s_mask[4 * lane + q]) : 0;
      }
      const int own = incl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      rows = __shfl_sync(0xffffffffu, incl, 31);
      for (int w = warp; w < words; w += kClusterWarps) {
        const int from = w >> 2;
        const int at = (w & 3) == 0 ? c[0] : (w & 3) == 1 ? c[1] : (w & 3) == 2 ? c[2] : c[3];
        const int before = __shfl_sync(0xffffffffu, incl - own + at, from);
        const unsigned b = s_mask[w];
        if ((b >> lane) & 1u) list[before + __popc(b & ((1u << lane) - 1u))] = 32 * w + lane;
      }
    }
    __syncthreads();
    const int all_warps = ctas * kClusterWarps;
    int ps = 0;  // log2 of a row's parts
    while ((2 << ps) * rows <= all_warps && (64 << ps) < m && ps < 5) ++ps;
    const int items = rows << ps;
    WideCand best{LLONG_MAX, 0, INT_MAX, INT_MAX, -1, -1};
    for (int w = rank * kClusterWarps + warp; w < items; w += all_warps) {
      const int row = list[w >> ps], part = w & ((1 << ps) - 1);
      const int64_t rr = NJ ? r[row] : 0;
      const int64_t *p = A.D + (row == f ? src_f : row) * n;
      const int col1 = lane + 32 * part, hop = 32 << ps;
      // Calls visit(col, distance) for this lane's columns of the row.
      auto sweep = [&](auto visit) {
        if (row == a) {
          for (int col = col1; col < m; col += hop)
            if (col != a) visit(col, du[col]);
          return;
        }
        constexpr int U = 16;
        for (int col0 = col1; col0 < m; col0 += hop * U) {
          int64_t d[U];
#pragma unroll
          for (int q = 0; q < U; ++q) d[q] = col0 + hop * q < m ? __ldcg(p + col0 + hop * q) : 0;
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const int col = col0 + hop * q;
            if (col < m && col != row && col != a && col != f) visit(col, d[q]);
          }
        }
        if (part == 0 && lane == 0 && a >= 0) visit(a, du[row]);
        if (part == 0 && lane == 1 && f < m && row != f) visit(f, __ldcg(p + src_f));
      };
      auto criterion = [&](int col, int64_t d) { return NJ ? m2 * d - rr - r[col] : d; };
      // The smallest criterion first, by selects (positions, read for every
      // new minimum of a lane, made the warp branch at most columns: 6,600 of
      // 16,500 cycles a join at 2,003 leaves); positions only where it is tied.
      WideCand rb{LLONG_MAX, 0, INT_MAX, INT_MAX, row, -1};
      bool tied = false;
      sweep([&](int col, int64_t d) {
        const int64_t c = criterion(col, d);
        const bool less = c < rb.c;
        tied = !less && (tied || c == rb.c);
        rb.c = less ? c : rb.c;
        rb.d = less ? d : rb.d;
        rb.sb = less ? col : rb.sb;
      });
      const int64_t least = warp_min(rb.c);
      const unsigned who = __ballot_sync(0xffffffffu, rb.c == least);
      int b = __ffs(who) - 1;
      if (__popc(who) > 1 || ((__ballot_sync(0xffffffffu, tied) >> b) & 1u)) {
        const int32_t pr = pos[row];
        sweep([&](int col, int64_t d) {
          if (criterion(col, d) != least) return;
          const int32_t pc = pos[col], lo = min(pr, pc), hi = max(pr, pc);
          if (lo < rb.lo || (lo == rb.lo && hi < rb.hi)) rb = WideCand{least, d, lo, hi, row, col};
        });
        b = best_lane(rb.c, rb.lo, rb.hi);
      }
      rb.c = least;
      rb.d = __shfl_sync(0xffffffffu, rb.d, b);
      rb.sb = __shfl_sync(0xffffffffu, rb.sb, b);
      if (w < kRefresh && lane < ctas) *cluster.map_shared_rank(&refresh[w], lane) = Refresh{rb.c, rb.d, row, rb.sb};
      if (items > kRefresh) {  // (the first joins: more rows than results kept)
        rb.lo = rb.sb < 0 ? INT_MAX : min(pos[row], pos[rb.sb]);
        rb.hi = rb.sb < 0 ? INT_MAX : max(pos[row], pos[rb.sb]);
        if (better_pair(best, rb.c, rb.lo, rb.hi)) best = rb;
      }
    }
    if (items > kRefresh) {
      if (lane == 0) s_warp[warp] = best;
      __syncthreads();
      if (warp == 0) {
        const WideCand w = s_warp[lane % kClusterWarps];
        const int b = best_lane(lane < kClusterWarps ? w.c : LLONG_MAX, w.lo, w.hi) % kClusterWarps;
        if (lane < ctas) *cluster.map_shared_rank(&s_cand[rank], lane) = s_warp[b];
      }
    }
    cluster.sync();  // barrier A

    // ---- 2. pick, read the joined rows, new bounds, update the tables ----
    WideCand pick{LLONG_MAX, 0, INT_MAX, INT_MAX, -1, -1};
    if (items > kRefresh) {
      const WideCand x = s_cand[lane % ctas];
      pick = s_cand[best_lane(lane < ctas ? x.c : LLONG_MAX, x.lo, x.hi) % ctas];
      if (!NJ && better_pair(pick, settled.c, settled.lo, settled.hi)) pick = settled;
    } else {
      if (!NJ && lane == 0) pick = settled;
      for (int e = lane; e < items; e += 32) {
        const Refresh x = refresh[e];
        if (x.near < 0 || x.c > pick.c) continue;
        const int32_t p = pos[x.row], q = pos[x.near], lo = min(p, q), hi = max(p, q);
        if (better_pair(pick, x.c, lo, hi))
          pick = WideCand{x.c, x.d, lo, hi, x.row, x.near};
      }
      const int b = best_lane(pick.c, pick.lo, pick.hi);
      pick.d = __shfl_sync(0xffffffffu, pick.d, b);
      pick.lo = __shfl_sync(0xffffffffu, pick.lo, b);
      pick.sa = __shfl_sync(0xffffffffu, pick.sa, b);
      pick.sb = __shfl_sync(0xffffffffu, pick.sb, b);
    }
    if (pick.sa < 0) {
      if (rank == 0 && tid == 0) A.st->error = 1;
      break;  // (the same for every CTA)
    }
    const int i = pos[pick.sa] == pick.lo ? pick.sa : pick.sb;
    const int j = i == pick.sa ? pick.sb : pick.sa;
    const int64_t dij = pick.d, si = size[i], sj = size[j];
    const int L = m - 1;
    const int na = i != L ? i : j, nf = na == i ? j : i;
    const bool move = nf != L;
    // The loads go out first: rows i and j (the first V slots of this thread),
    // row L's entry for step 3, and what the record of the join, written at
    // the end, needs (the children's heights: this thread's own records, or
    // those of the joins before this launch).
    const int64_t *pi = A.D + i * n, *pj = A.D + j * n;
    constexpr int V = 8;
    int64_t di[V], dj[V];
    auto load = [&](int k0) {
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const int k = k0 + q * kClusterThreads;
        di[q] = k < m ? __ldcg(pi + k) : 0;
        dj[q] = k < m ? __ldcg(pj + k) : 0;
      }
    };
    load(tid);
    const int k3 = rank * kClusterThreads + tid;
    const int64_t dL = k3 < m ? __ldcg(A.D + L * n + k3) : 0;
    const bool recorder = rank == 0 && tid == 0;
    int64_t hi_ = 0, hj_ = 0;
    int32_t left = 0, right = 0;
    if (recorder) {
      left = node[i];
      right = node[j];
      if (NJ) {
        hi_ = r[i];
        hj_ = r[j];
      } else {
        if (left >= n) hi_ = A.out[left - n].height;
        if (right >= n) hj_ = A.out[right - n].height;
      }
    }
    // New bounds: the least of each row's parts (a power of two of lanes).
    for (int e0 = warp * 32; e0 < min(items, kRefresh); e0 += kClusterThreads) {
      const int e = e0 + lane;
      Refresh x{LLONG_MAX, 0, 0, -1};
      if (e < min(items, kRefresh)) x = refresh[e];
      for (int o = 1; o < (1 << ps); o <<= 1) {
        const int64_t c = __shfl_xor_sync(0xffffffffu, x.c, o), d = __shfl_xor_sync(0xffffffffu, x.d, o);
        const int32_t nr = __shfl_xor_sync(0xffffffffu, x.near, o);
        bool take = c < x.c;
        if (c == x.c && nr >= 0 && x.near >= 0) {  // (tied parts: the smaller positions)
          const int32_t p = pos[x.row], q = pos[x.near], u = pos[nr];
          const int32_t lo = min(p, q), lo2 = min(p, u);
          take = lo2 < lo || (lo2 == lo && max(p, u) < max(p, q));
        }
        if (take) {
          x.c = c;
          x.d = d;
          x.near = nr;
        }
      }
      if (e < min(items, kRefresh) && (e & ((1 << ps) - 1)) == 0) {
        bound[x.row] = x.c;
        near[x.row] = x.near;
        near_d[x.row] = x.d;
      }
    }
    const uint32_t sum_size = uint32_t(si + sj);  // (at most 65,535)
    uint64_t inv = 0;
    if (!NJ) {
      // floor((2^64 - 1) / sum_size) by three 32-bit divisions.
      const uint32_t q0 = 0xffffffffu / sum_size, r0 = 0xffffffffu - q0 * sum_size;
      const uint32_t x1 = (r0 << 16) | 0xffffu, q1 = x1 / sum_size, r1 = x1 - q1 * sum_size;
      const uint32_t x2 = (r1 << 16) | 0xffffu, q2 = x2 / sum_size;
      inv = (uint64_t(q0) << 32) | (uint64_t(q1) << 16) | q2;
    }
    __syncthreads();
    int64_t rsum = 0, dlo = LLONG_MAX, dhi = dmax;
    for (int k0 = tid; k0 < m; k0 += V * kClusterThreads) {
      if (k0 != tid) load(k0);
#pragma unroll
      for (int q = 0; q < V; ++q) {
        const int k = k0 + q * kClusterThreads;
        if (k >= m) break;
        if (k == i || k == j) continue;
        const int64_t v = NJ ? (di[q] + dj[q] - dij) >> 1 : floor_div_by(si * di[q] + sj * dj[q], sum_size, inv);
        du[k] = v;
        if (NJ) {
          const int64_t delta = di[q] + dj[q] - v;
          r[k] -= delta;
          bound[k] += delta;
          rsum += v;
          dlo = delta < dlo ? delta : dlo;
          dhi = v > dhi ? v : dhi;
        }
      }
    }
    cluster.barrier_arrive();  // barrier B
    if (NJ) {
      block_sum_min_max(rsum, dlo, dhi);
      dmax = dhi;
    }
    const int64_t ru = rsum, drift = NJ ? dlo - dmax : 0;
    int64_t known = LLONG_MAX;
    WideCand mine{LLONG_MAX, 0, INT_MAX, INT_MAX, -1, -1}, joined = mine;  // UPGMA: settled rows, row na
    for (int k = tid; k < m; k += kClusterThreads) {
      if (k == i || k == j) continue;
      const int64_t v = du[k];
      int32_t x = near[k];
      if constexpr (NJ) {
        const int64_t qn = (m2 - 1) * v - r[k] - ru, lb = bound[k] + drift;
        bound[k] = qn < lb ? qn : lb;
        if (qn <= lb || x == i || x == j) {
          near[k] = na;
          near_d[k] = v;
          known = qn < known ? qn : known;
        } else if (x >= 0) {
          const int64_t q = (m2 - 1) * near_d[k] - r[k] - r[x];
          known = q < known ? q : known;
          if (x == L) near[k] = nf;  // (L is not i or j here: it moves)
        }
      } else {
        // The new pair (k, na): below the bound it settles the row; tied with
        // the neighbour of a settled row, the smaller positions stay.  A row
        // that loses its neighbour is open (ties of it are not known).
        const int32_t pk = pos[k], lo = min(pk, pick.lo), hi = max(pk, pick.lo);
        const int64_t lb = bound[k];
        bool is_settled = x >= 0 && x != i && x != j && near_d[k] == lb;
        if (v < lb) {
          bound[k] = near_d[k] = v;
          x = na;
          is_settled = true;
        } else if (is_settled && v == lb) {
          const int32_t px = pos[x], xlo = min(pk, px), xhi = max(pk, px);
          if (lo < xlo || (lo == xlo && hi < xhi)) x = na;
        } else if (!is_settled) {
          x = -1;
        }
        near[k] = x == L ? nf : x;
        known = v < known ? v : known;
        const int32_t slot = k == L ? nf : k;
        if (better_pair(joined, v, lo, hi)) joined = WideCand{v, v, lo, hi, na, slot};
        if (is_settled) {
          const int32_t px = x == na ? pick.lo : pos[x];
          const int64_t c = bound[k];
          known = c < known ? c : known;
          if (better_pair(mine, c, min(pk, px), max(pk, px)))
            mine = WideCand{c, c, min(pk, px), max(pk, px), slot, x == L ? nf : x};
        }
      }
    }
    if (!NJ) {
      int b = best_lane(mine.c, mine.lo, mine.hi);
      if (lane == b) s_warp[warp] = mine;
      b = best_lane(joined.c, joined.lo, joined.hi);
      if (lane == b) s_joined[warp] = joined;
    }
    ub = block_min(known, 3);
    if (!NJ) {
      const WideCand x = s_warp[lane % kClusterWarps], y = s_joined[lane % kClusterWarps];
      settled = s_warp[best_lane(lane < kClusterWarps ? x.c : LLONG_MAX, x.lo, x.hi) % kClusterWarps];
      joined = s_joined[best_lane(lane < kClusterWarps ? y.c : LLONG_MAX, y.lo, y.hi) % kClusterWarps];
    }
    if (tid == 0) {
      if (move) {
        r[nf] = r[L];
        pos[nf] = pos[L];
        node[nf] = node[L];
        size[nf] = size[L];
        du[nf] = du[L];
        bound[nf] = bound[L];
        near[nf] = near[L];
        near_d[nf] = near_d[L];
      }
      r[na] = ru;
      node[na] = int32_t(n + t);
      size[na] = int32_t(si + sj);
      pos[na] = pick.lo;
      bound[na] = NJ ? kUnknown : joined.c;  // (NJ: scanned next, from du)
      near[na] = NJ ? -1 : joined.sb;
      near_d[na] = joined.d;
    }
    cluster.barrier_wait();  // barrier B
    __syncthreads();
    // ---- 3. write this CTA's share of the new distances ----
    for (int k = k3; k < m - 1; k += ctas * kClusterThreads) {
      if (k == na) continue;
      A.D[na * n + k] = du[k];
      A.D[k * n + na] = du[k];
      if (move && k != nf) {
        const int64_t v = k == k3 ? dL : __ldcg(A.D + L * n + k);
        A.D[nf * n + k] = v;
        A.D[k * n + nf] = v;
      }
    }
    if (recorder) {
      tsq_tree_node o;
      o.left = left;
      o.right = right;
      o.size = int32_t(si + sj);
      o.pos = pick.lo;
      o.dist = dij;
      if (NJ) {
        o.height = 0;
        o.left_length = m > 2 ? floor_div(m2 * dij + hi_ - hj_, 2 * m2) : (dij >> 1);
        o.right_length = dij - o.left_length;
      } else {
        const int64_t h = dij >> 1;
        o.height = h;
        o.left_length = h - hi_;
        o.right_length = h - hj_;
      }
      A.out[t] = o;
    }
    a = na;
    f = move ? nf : m;  // (no row f: every slot is below m - 1 from now on)
    src_f = L;
  }
  if (rank == 0 && tid == 0 && !A.st->error) {
    A.st->m = 1;
    A.st->t = int32_t(n) - 1;
  }
}

__device__ __forceinline__ int64_t identity_distance(int32_t n_ident, int32_t n_cols) {
  if (n_cols <= 0) return int64_t(1) << 32;
  return int64_t((uint64_t(uint32_t(n_cols - n_ident)) << 32) / uint64_t(uint32_t(n_cols)));
}

// D from identities of the unordered pairs (i < j) in row-major order; the
// identities sit `stride` int32 apart (1 for plain arrays, 8 for ResultDev
// records), with the pair status `status_off` ints after n_ident (or none).
__global__ void tree_init_kernel(int64_t *D, int32_t n, const int32_t *ident, const int32_t *cols, int32_t stride,
                                 const int32_t *status, TreeState *st) {
  const int32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t i = blockIdx.y;
  if (j >= n) return;
  if (i == j) {
    D[int64_t(i) * n + j] = 0;
    return;
  }
  const int32_t lo = min(i, j), hi = max(i, j);
  const int64_t k = int64_t(lo) * (2 * int64_t(n) - lo - 1) / 2 + (hi - lo - 1);
  const int32_t ni = ident[k * stride], nc = cols[k * stride];
  if ((status && status[k * stride] != 0) || nc < 0 || ni < 0 || ni > nc) st->error = 2;
  D[int64_t(i) * n + j] = identity_distance(ni, nc);
}

__global__ void tree_slots_kernel(const int64_t *D, int32_t n, int64_t *r, int64_t *height, int32_t *pos,
                                  int32_t *node, int32_t *size, TreeState *st) {
  const int32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w == 0 && lane == 0) {
    st->m = n;
    st->t = 0;
    st->ticket = 0u;
  }
  if (w >= n) return;
  int64_t s = 0;
  for (int32_t k = lane; k < n; k += 32)
    if (k != w) s += D[int64_t(w) * n + k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    r[w] = s;
    height[w] = 0;
    pos[w] = w;
    node[w] = w;
    size[w] = 1;
  }
}

__global__ void tree_error_reset_kernel(TreeState *st) { st->error = 0; }

int sm_count() {
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// CTAs of the join cluster on the current device: 16 where a cluster of that
// size can be resident, else 8, else none (0: two launches per join).
int tree_cluster_ctas() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  static std::mutex mu;
  static std::map<int, int> known;
  std::lock_guard<std::mutex> g(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  int best = 0;
  for (int ctas : {kMaxClusterCtas, 8}) {
    bool fits = true;
    for (auto k : {tree_cluster_kernel<true>, tree_cluster_kernel<false>}) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(unsigned(ctas));
      cfg.blockDim = dim3(kClusterThreads);
      cfg.dynamicSmemBytes = kRefresh * sizeof(Refresh) + size_t(kClusterLeaves) * kSlotBytes;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = unsigned(ctas);
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      fits = fits && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
             cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cfg.dynamicSmemBytes)) ==
                 cudaSuccess &&
             cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters > 0;
    }
    if (fits) {
      best = ctas;
      break;
    }
  }
  cudaGetLastError();  // (a size that does not fit is not an error)
  known[dev] = best;
  return best;
}

struct TreeBufs {
  DevBuf D, small, partial, out, ids;
  cudaStream_t stream = nullptr;
  int dev = -1;
  ~TreeBufs() {
    if (stream) cudaStreamDestroy(stream);
  }
};

constexpr int32_t kMaxTreeLeaves = 65535;  // one grid row per leaf in tree_init_kernel

// Sizes the buffers for n leaves and fills TreeArgs.
cudaError_t tree_prepare(TreeBufs &b, int32_t n, TreeArgs *A) {
  const size_t nn = size_t(n) * size_t(n);
  cudaError_t e = b.D.ensure(nn * 8);
  const size_t small = size_t(n) * (8 + 8 + 4 + 4 + 4) + sizeof(TreeState) + 64;
  if (e == cudaSuccess) e = b.small.ensure(small);
  const int parts = 4 * sm_count();
  if (e == cudaSuccess) e = b.partial.ensure(size_t(parts) * sizeof(Cand));
  if (e == cudaSuccess) e = b.out.ensure(size_t(n > 1 ? n - 1 : 1) * sizeof(tsq_tree_node));
  if (e != cudaSuccess) return e;
  char *p = b.small.as<char>();
  A->D = b.D.as<int64_t>();
  A->r = reinterpret_cast<int64_t *>(p);
  A->height = A->r + n;
  A->pos = reinterpret_cast<int32_t *>(A->height + n);
  A->node = A->pos + n;
  A->size = A->node + n;
  A->st = reinterpret_cast<TreeState *>((reinterpret_cast<uintptr_t>(A->size + n) + 15) & ~uintptr_t(15));
  A->partial = b.partial.as<Cand>();
  A->out = b.out.as<tsq_tree_node>();
  A->n = n;
  return cudaSuccess;
}

// Row sums, slot tables, then the n-1 joins; copies the joins to `out`.
int tree_run(const TreeArgs &A, int32_t method, cudaStream_t s, tsq_tree_node *out) {
  const int32_t n = A.n;
  tree_slots_kernel<<<(n + 7) / 8, 256, 0, s>>>(A.D, n, A.r, A.height, A.pos, A.node, A.size, A.st);
  const int parts = 4 * sm_count();
  const bool nj = method == TSQ_TREE_NJ;
  const int ctas = tree_cluster_ctas();
  int32_t t = 0;
  for (; t < n - 1 && (ctas == 0 || n - t > kClusterLeaves); ++t) {
    const int32_t m = n - t;
    const int blocks = std::max(1, std::min(parts, m / 2));
    const int jblocks = std::max(1, std::min(parts, (m + kTreeThreads - 1) / kTreeThreads));
    if (nj) {
      tree_scan_kernel<true><<<blocks, kTreeThreads, 0, s>>>(A, m, t);
      tree_join_kernel<true><<<jblocks, kTreeThreads, 0, s>>>(A, m, t);
    } else {
      tree_scan_kernel<false><<<blocks, kTreeThreads, 0, s>>>(A, m, t);
      tree_join_kernel<false><<<jblocks, kTreeThreads, 0, s>>>(A, m, t);
    }
  }
  if (t < n - 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(ctas));
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = kRefresh * sizeof(Refresh) + size_t(n - t) * kSlotBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(ctas);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = nj ? cudaLaunchKernelEx(&cfg, tree_cluster_kernel<true>, A, n - t, t)
                             : cudaLaunchKernelEx(&cfg, tree_cluster_kernel<false>, A, n - t, t);
    if (e != cudaSuccess) return cuda_status(e);
  }
  cudaError_t e = cudaGetLastError();
  TreeState st{};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&st, A.st, sizeof(st), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && n > 1)
    e = cudaMemcpyAsync(out, A.out, sizeof(tsq_tree_node) * size_t(n - 1), cudaMemcpyDeviceToHost, s);
  const cudaError_t sy = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = sy;
  if (e != cudaSuccess) return cuda_status(e);
  if (st.error == 2) return TSQ_E_INVALID_ARG;
  if (st.error != 0 || st.m != 1 || st.t != n - 1) return TSQ_E_CUDA;
  return TSQ_OK;
}

TreeBufs &tree_cache(int *rc) {
  thread_local TreeBufs c;
  int dev = 0;
  *rc = TSQ_OK;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    *rc = TSQ_E_CUDA;
    return c;
  }
  if (c.dev != dev) {
    c.D.release();
    c.small.release();
    c.partial.release();
    c.out.release();
    c.ids.release();
    if (c.stream) cudaStreamDestroy(c.stream);
    c.stream = nullptr;
    if (cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking) != cudaSuccess) {
      *rc = TSQ_E_CUDA;
      return c;
    }
    c.dev = dev;
  }
  return c;
}

bool bad_method(int32_t method) { return method != TSQ_TREE_UPGMA && method != TSQ_TREE_NJ; }

}  // namespace
}  // namespace tsq

extern "C" {

int tsq_guide_tree_dist(int32_t n, const int64_t *dist, int32_t method, tsq_tree_node *out) {
  if (n < 1 || n > tsq::kMaxTreeLeaves || !dist || tsq::bad_method(method) || (n > 1 && !out))
    return TSQ_E_INVALID_ARG;
  if (n == 1) return TSQ_OK;
  for (int32_t i = 0; i < n; ++i)
    for (int32_t j = i + 1; j < n; ++j)
      if (dist[int64_t(i) * n + j] != dist[int64_t(j) * n + i]) return TSQ_E_INVALID_ARG;
  try {
    int rc = TSQ_OK;
    tsq::TreeBufs &b = tsq::tree_cache(&rc);
    if (rc) return rc;
    tsq::TreeArgs A;
    cudaError_t e = tsq::tree_prepare(b, n, &A);
    if (e == cudaSuccess) e = cudaMemcpyAsync(A.D, dist, size_t(n) * size_t(n) * 8, cudaMemcpyHostToDevice, b.stream);
    if (e == cudaSuccess) {
      tsq::tree_error_reset_kernel<<<1, 1, 0, b.stream>>>(A.st);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return tsq::cuda_status(e);
    return tsq::tree_run(A, method, b.stream, out);
  } catch (const std::bad_alloc &) {
    return TSQ_E_NOMEM;
  }
}

int tsq_guide_tree(int32_t n, const int32_t *n_ident, const int32_t *n_cols, int32_t method, tsq_tree_node *out) {
  if (n < 1 || n > tsq::kMaxTreeLeaves || tsq::bad_method(method) || (n > 1 && (!out || !n_ident || !n_cols)))
    return TSQ_E_INVALID_ARG;
  if (n == 1) return TSQ_OK;
  try {
    int rc = TSQ_OK;
    tsq::TreeBufs &b = tsq::tree_cache(&rc);
    if (rc) return rc;
    tsq::TreeArgs A;
    const int64_t npairs = int64_t(n) * (n - 1) / 2;
    cudaError_t e = tsq::tree_prepare(b, n, &A);
    if (e == cudaSuccess) e = b.ids.ensure(size_t(npairs) * 8);
    int32_t *d_ident = b.ids.as<int32_t>(), *d_cols = d_ident + npairs;
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(d_ident, n_ident, size_t(npairs) * 4, cudaMemcpyHostToDevice, b.stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_cols, n_cols, size_t(npairs) * 4, cudaMemcpyHostToDevice, b.stream);
    if (e == cudaSuccess) {
      tsq::tree_error_reset_kernel<<<1, 1, 0, b.stream>>>(A.st);
      tsq::tree_init_kernel<<<dim3((n + 255) / 256, n), 256, 0, b.stream>>>(A.D, n, d_ident, d_cols, 1, nullptr,
                                                                            A.st);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return tsq::cuda_status(e);
    return tsq::tree_run(A, method, b.stream, out);
  } catch (const std::bad_alloc &) {
    return TSQ_E_NOMEM;
  }
}

int tsq_batch_guide_tree(tsq_batch *bt, int32_t n, int32_t method, tsq_tree_node *out) {
  if (!bt || n < 1 || n > tsq::kMaxTreeLeaves || tsq::bad_method(method) || (n > 1 && !out))
    return TSQ_E_INVALID_ARG;
  if (bt->out_mode == tsq::kOutScore || int64_t(n) * (n - 1) / 2 != bt->n || !bt->has_run) return TSQ_E_INVALID_ARG;
  if (n == 1) return TSQ_OK;
  // The batch must be the all-vs-all of n sequences in row-major pair order:
  // every pair (i, j) reads sequence i as a and sequence j as b.
  {
    std::vector<int64_t> off(static_cast<size_t>(n));
    std::vector<int32_t> len(static_cast<size_t>(n));
    for (int32_t s = 0; s + 1 < n; ++s) {
      const int64_t k = int64_t(s) * (2 * int64_t(n) - s - 1) / 2;  // pair (s, s + 1)
      off[size_t(s)] = bt->pairs_h[size_t(k)].a_off;
      len[size_t(s)] = bt->pairs_h[size_t(k)].a_len;
    }
    off[size_t(n - 1)] = bt->pairs_h[size_t(n - 2)].b_off;  // pair (0, n - 1)
    len[size_t(n - 1)] = bt->pairs_h[size_t(n - 2)].b_len;
    int64_t k = 0;
    for (int32_t i = 0; i < n; ++i)
      for (int32_t j = i + 1; j < n; ++j, ++k) {
        const tsq::PairDev &p = bt->pairs_h[size_t(k)];
        if (p.a_off != off[size_t(i)] || p.a_len != len[size_t(i)] || p.b_off != off[size_t(j)] ||
            p.b_len != len[size_t(j)])
          return TSQ_E_INVALID_ARG;
      }
  }
  try {
    if (cudaSetDevice(bt->device) != cudaSuccess) return TSQ_E_CUDA;
    int rc = TSQ_OK;
    tsq::TreeBufs &b = tsq::tree_cache(&rc);
    if (rc) return rc;
    tsq::TreeArgs A;
    cudaError_t e = tsq::tree_prepare(b, n, &A);
    const int32_t *res = bt->res.as<int32_t>();
    if (e == cudaSuccess) {
      // The distances are built on the batch's stream, after its run.
      tsq::tree_error_reset_kernel<<<1, 1, 0, bt->stream>>>(A.st);
      tsq::tree_init_kernel<<<dim3((n + 255) / 256, n), 256, 0, bt->stream>>>(
          A.D, n, res + offsetof(tsq::ResultDev, n_ident) / 4, res + offsetof(tsq::ResultDev, n_cols) / 4,
          int32_t(sizeof(tsq::ResultDev) / 4), res + offsetof(tsq::ResultDev, status) / 4, A.st);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return tsq::cuda_status(e);
    return tsq::tree_run(A, method, bt->stream, out);
  } catch (const std::bad_alloc &) {
    return TSQ_E_NOMEM;
  }
}

}  // extern "C"
