// walk_kernel.cu -- traceback walker and residue encoder.
//
// The walker follows the 4-bit direction planes written by the fill from the
// end cell back to the start, exactly as the CPU oracle's walk does (state
// machine over H, E and F; E and F runs end where the "opened" bit is set;
// global rows/columns 0 are single gap runs; local stops on a STOP cell or
// row/column 0).  It emits the two gapped rows backwards into the pair's
// output slot, so the aligned strings end at slot + cap and start at
// slot + cap - n_cols, and records identity, column count and the begin
// coordinates.
#include <algorithm>

#include "tsq_internal.h"

namespace tsq {
namespace {

// The walk of one pair, from its end cell back to its start, through a
// plane reader and two sequence readers.  Every lane of the pair's warp runs
// it with the same values (warp-uniform branches); only `writer` (lane 0)
// stores, except in a run of diagonal moves, where lane k writes the k-th
// column of the run.
template <class Plane, class Seq>
__device__ __forceinline__ void walk_pair(const WalkArgs &A, const PairDev &pr, ResultDev &res, Plane &pl, Seq &a,
                                          Seq &b, char *out_a, char *out_b, int64_t cap, int lane) {
  const bool emit = A.emit != 0, lead = lane == 0, writer = lead && emit;
  const int m = pr.a_len, n = pr.b_len;
  int i, j;
  if (A.local) {
    if (res.score <= 0) {
      if (lead) {
        res.a_begin = res.a_end = res.b_begin = res.b_end = 0;
        res.n_ident = res.n_cols = 0;
      }
      return;
    }
    i = res.a_end;
    j = res.b_end;
  } else {
    i = m;
    j = n;
  }
  if (i > 0) pl.set_row(i);
  int state = 0;  // 0 = H, 1 = E, 2 = F
  int64_t L = 0;
  int ident = 0;
  for (;;) {
    if (L >= cap && (i > 0 || j > 0)) {  // cannot happen with valid planes
      if (lead) res.status = TSQ_E_CUDA;
      return;
    }
    if (state == 0) {
      if (A.local) {
        if (i == 0 || j == 0 || pl.dir(j) == kDirStop) break;
      } else if (i == 0 && j == 0) {
        break;
      }
      if (i > 0 && j > 0) {
        // A run of diagonal moves at once: lane k tests the cell k steps back
        // along the diagonal, inside the plane window loaded around the
        // current cell (a cell outside it ends the run); the leading run of
        // diagonal cells becomes p aligned columns, lane k writing the k-th.
        (void)pl.nib(j);
        const uint32_t dm = pl.diag_mask(i, j);
        const int p = dm == 0xffffffffu ? 32 : __ffs(~dm) - 1;
        if (p > 1) {
          a.cover(i - 1);
          b.cover(j - 1);
          uint8_t ca = 0, cb = 0;
          if (lane < p) {
            ca = a.get(i - 1 - lane);
            cb = b.get(j - 1 - lane);
            if (emit) {
              out_a[cap - L - 1 - lane] = char(ca);
              out_b[cap - L - 1 - lane] = char(cb);
            }
          }
          ident += __popc(__ballot_sync(0xffffffffu, lane < p && ca == cb));
          L += p;
          i -= p;
          j -= p;
          if (i > 0) pl.set_row(i);
          continue;
        }
      }
      if (i == 0) {  // global top row: one horizontal gap run
        ++L;
        const char cb = char(b.at(j - 1));
        if (writer) {
          out_a[cap - L] = '-';
          out_b[cap - L] = cb;
        }
        --j;
        continue;
      }
      if (j == 0) {  // global left column: one vertical gap run
        ++L;
        const char ca = char(a.at(i - 1));
        if (writer) {
          out_a[cap - L] = ca;
          out_b[cap - L] = '-';
        }
        --i;
        if (i > 0) pl.up();
        continue;
      }
      const int hd = pl.dir(j);
      if (hd == kDirDiag) {
        ++L;
        const uint8_t ca = a.at(i - 1), cb = b.at(j - 1);
        if (writer) {
          out_a[cap - L] = char(ca);
          out_b[cap - L] = char(cb);
        }
        ident += ca == cb;
        --i;
        --j;
        if (i > 0) pl.up();
      } else {
        state = hd;
      }
    } else if (state == 1) {
      // An E run always ends inside the matrix (E(i,0) is minus infinity);
      // if the planes say otherwise, stop instead of leaving the matrix.
      if (j <= 0 || i <= 0) {
        if (lead) res.status = TSQ_E_CUDA;
        return;
      }
      const int d = pl.nib(j);
      ++L;
      const char cb = char(b.at(j - 1));
      if (writer) {
        out_a[cap - L] = '-';
        out_b[cap - L] = cb;
      }
      --j;
      if (d & 4) state = 0;
    } else {
      if (i <= 0 || j <= 0) {
        if (lead) res.status = TSQ_E_CUDA;
        return;
      }
      const int d = pl.nib(j);
      ++L;
      const char ca = char(a.at(i - 1));
      if (writer) {
        out_a[cap - L] = ca;
        out_b[cap - L] = '-';
      }
      --i;
      if (i > 0) pl.up();
      if (d & 8) state = 0;
    }
  }
  if (!lead) return;
  if (emit || !A.local) {
    res.a_begin = i;
    res.b_begin = j;
  }
  if (!A.local) {
    res.a_end = m;
    res.b_end = n;
  }
  res.n_cols = int32_t(L);
  res.n_ident = ident;
}

// One warp per pair, every lane running the pair's walk with the same
// values, so a window refill costs the warp one coalesced load per lane and
// the warp waits only for its own pair's refills.  (A thread per pair made
// each warp wait for all 32 of its pairs' refills in turn: 0.77 against
// 0.14 ms on 2,016 protein pairs, 18.3 against 3.2 ms on 32 long DNA pairs,
// 3.8 against 3.6 ms on 100,000 pairs.)
constexpr int kWarpWalkWarps = 4;
// Pairs up to which the walks leave most of the GPU idle (one warp each on
// 152 SMs).
constexpr int kWideWalks = 1024;

// The planes of one pair, read through a window in shared memory.  Cells are
// placed by their global lane g = (i - 1) / R (R rows per lane) and their
// global step q = j - 1 + g, across bands; a word holds eight cells, U = 8 / R
// steps.  The window holds WS words of steps x WL lanes: a diagonal run of c
// cells needs c / R + 1 lanes and (c + c / R) / U + 1 words.
template <int R, int WS, int WL>
struct WarpPlane {
  static constexpr int kWords = WS * WL;
  static constexpr int kRShift = R == 8 ? 3 : 2, kUShift = 3 - kRShift;
  const uint32_t *words;
  uint32_t *win;  // kWords words of this warp
  int row_words;  // words of a band per lane
  int gshift, lane;
  uint32_t diag_bits;  // bits that are 0 where H is the diagonal's: 3 local, 1 global
  int g = 0, r = 0;
  int wg = -1, ws = -1;
  static __device__ int band_words(int n, int G) { return (n + G - 1 + (1 << kUShift) - 1) >> kUShift; }
  __device__ void set_row(int i) {
    g = (i - 1) >> kRShift;
    r = (i - 1) & (R - 1);
  }
  __device__ void up() {
    if (--r < 0) {
      r = R - 1;
      --g;
    }
  }
  // The nibble of row `row` at step q in its word: the row's own (R = 8), or
  // the rows of U steps from the top down.
  static __device__ int shift_of(int q, int row) {
    return R == 8 ? 4 * row : 4 * (7 - ((q & ((1 << kUShift) - 1)) * R + row));
  }
  // Words s-WS+1..s of lanes g-WL+1..g (clamped into the planes).
  __device__ void refill(int s) {
    wg = g;
    ws = s;
    uint32_t v[(kWords + 31) / 32];
#pragma unroll
    for (int q = 0; q < (kWords + 31) / 32; ++q) {
      const int w = lane + 32 * q;
      const int gg = max(g - w % WL, 0);
      const int band = gg >> gshift, t = gg & ((1 << gshift) - 1);
      const int ss = min(max(s - w / WL - ((band << gshift) >> kUShift), 0), row_words - 1);
      v[q] = __ldg(words + ((((int64_t)band * row_words + ss) << gshift) + t));
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < (kWords + 31) / 32; ++q)
      if (kWords % 32 == 0 || lane + 32 * q < kWords) win[lane + 32 * q] = v[q];
    __syncwarp();
  }
  __device__ int nib(int j) {
    const int q = j - 1 + g, s = q >> kUShift;
    if (g > wg || g <= wg - WL || s > ws || s <= ws - WS) refill(s);
    return int(win[(ws - s) * WL + (wg - g)] >> shift_of(q, r)) & 15;
  }
  // Where H of the cell comes from.
  __device__ int dir(int j) {
    const int v = nib(j);
    if ((uint32_t(v) & diag_bits) == 0u) return kDirDiag;
    return diag_bits == 3u ? v & 3 : (v & 2 ? kDirF : kDirE);
  }
  // Lanes whose cell (i - lane, j - lane) lies inside the matrix and the
  // current window and takes H from the diagonal.
  __device__ uint32_t diag_mask(int i, int j) const {
    const int ik = i - lane, jk = j - lane;
    bool d = false;
    if (ik >= 1 && jk >= 1) {
      const int gk = (ik - 1) >> kRShift, rk = (ik - 1) & (R - 1);
      const int q = jk - 1 + gk, sk = q >> kUShift;
      if (gk > wg - WL && sk > ws - WS)
        d = ((win[(ws - sk) * WL + (wg - gk)] >> shift_of(q, rk)) & diag_bits) == 0u;
    }
    return __ballot_sync(0xffffffffu, d);
  }
  // Lanes whose cell (i, j - lane) (E) or (i - lane, j) (F) lies inside the
  // matrix and the current window and extends its gap.
  template <bool IN_ROW>
  __device__ uint32_t gap_mask(int i, int j) const {
    const int ik = IN_ROW ? i : i - lane, jk = IN_ROW ? j - lane : j;
    bool d = false;
    if (ik >= 1 && jk >= 1) {
      const int gk = (ik - 1) >> kRShift, rk = (ik - 1) & (R - 1);
      const int q = jk - 1 + gk, sk = q >> kUShift;
      if (gk > wg - WL && sk > ws - WS)
        d = ((win[(ws - sk) * WL + (wg - gk)] >> shift_of(q, rk)) & (IN_ROW ? 4u : 8u)) == 0u;
    }
    return __ballot_sync(0xffffffffu, d);
  }
};

// One sequence read backwards through a shared window of WIN residues.
template <int WIN>
struct WarpSeq {
  const uint8_t *base;
  int len;
  uint8_t *win;
  int lane;
  int lo = 1 << 30;
  // The window ending at idx.
  __device__ void refill_to(int idx) {
    lo = max(0, idx - WIN + 1);
    uint8_t v[WIN / 32];
#pragma unroll
    for (int q = 0; q < WIN / 32; ++q) {
      const int k = lo + lane + 32 * q;
      v[q] = k < len ? base[k] : uint8_t(0);
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < WIN / 32; ++q) win[lane + 32 * q] = v[q];
    __syncwarp();
  }
  __device__ uint8_t at(int idx) {
    if (idx < lo || idx >= lo + WIN) refill_to(idx);
    return win[idx - lo];
  }
  // Makes residues idx-31..idx (those >= 0) readable with get().
  __device__ void cover(int idx) {
    if (max(0, idx - 31) < lo || idx >= lo + WIN) refill_to(idx);
  }
  __device__ uint8_t get(int idx) const { return win[idx - lo]; }
};

template <int R, int WS, int WL, int WIN>
__device__ __forceinline__ void walk_one(const WalkArgs &A, int p, uint32_t *s_plane, uint8_t (*s_seq)[WIN], int lane) {
  using Plane = WarpPlane<R, WS, WL>;
  const PairDev pr = A.pairs[p];
  ResultDev &res = A.res[p];
  WarpSeq<WIN> a{A.seqs + pr.a_off, pr.a_len, s_seq[0], lane}, b{A.seqs + pr.b_off, pr.b_len, s_seq[1], lane};
  const int64_t cap = (int64_t)pr.a_len + pr.b_len;
  char *out_a = A.emit ? A.aln + A.aln_off[p] : nullptr;
  const int G = A.shape_G[p];
  Plane pl{reinterpret_cast<const uint32_t *>(A.planes + A.plane_off[p]), s_plane,
           Plane::band_words(pr.b_len, G), 31 - __clz(G), lane, A.local ? 3u : 1u};
  walk_pair(A, pr, res, pl, a, b, out_a, out_a + cap, cap, lane);
}

// WIDE: windows of about 48 diagonal cells and 512 residues instead of 24
// and 128.  A refill is one memory latency whatever its size, so few pairs,
// whose walks are a chain of refills on an idle GPU, take the wide ones; many
// pairs, whose refills overlap, the narrow ones, which read less.
template <bool WIDE>
__global__ void __launch_bounds__(kWarpWalkWarps * 32) walk_warp_kernel(const WalkArgs A) {
  constexpr int WIN = WIDE ? 512 : 128;
  constexpr int kWords = WIDE ? 576 : 182;
  __shared__ uint32_t s_plane[kWarpWalkWarps][kWords];
  __shared__ uint8_t s_seq[kWarpWalkWarps][2][WIN];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = blockIdx.x * kWarpWalkWarps + w;
  if (k >= A.n_tasks || (k >= A.skip_begin && k < A.skip_end)) return;
  const int p = A.tasks[k];
  if (A.res[p].status != TSQ_OK) return;
  const int R = A.shape_R[p];
  if constexpr (WIDE) {
    static_assert(64 * 9 <= kWords && 32 * 14 <= kWords, "windows fit");
    if (R == 4)
      walk_one<4, 32, 14, WIN>(A, p, s_plane[w], s_seq[w], lane);
    else
      walk_one<8, 64, 9, WIN>(A, p, s_plane[w], s_seq[w], lane);
  } else {
    static_assert(32 * 4 <= kWords && 20 * 9 <= kWords, "windows fit");
    if (R == 4)
      walk_one<4, 20, 9, WIN>(A, p, s_plane[w], s_seq[w], lane);
    else
      walk_one<8, 32, 4, WIN>(A, p, s_plane[w], s_seq[w], lane);
  }
}

// ---- one pair by many warps ---------------------------------------------
//
// A walk is a chain of dependent steps, about 50 ns a column on an idle GPU.
// For the pairs of the strip fill, few and long, the rows are cut into
// segments, one per warp of a block.  All warps walk their segment at once: the
// lowest from the true end cell, the others from a guessed cell of their
// lowest row (on the line from the end cell to the start).  Traceback paths that
// start near each other meet after a few cells and are one from there on, so
// what a warp walked is the true path but for its beginning.  Then every
// segment whose true entry -- the cell and state where the path of the segment
// below leaves it -- is not the one it started from walks again from there, until it
// meets what it recorded; rounds go on until every segment's entry is what
// the one below hands it.  The lowest segment is exact at once, and each round
// makes at least one more so: at most as many rounds as segments, the time of
// the plain walk, whatever the guesses; two or three where the sequences are
// related.  Every cell is a cell of the true path in the end, whichever way.
//
// A row's record: the column and state in which the path arrives in it, and
// how it leaves (diagonal, up, or not at all): its columns follow from that
// and the next row's arrival, so the gapped rows are written afterwards by all
// warps at offsets from a sum over them.
// One 20 kb pair (DNA, 10 % substitutions, 2 % indels) 1.10 -> 0.10 ms, 23 pairs of
// 10 to 50 kb 2.60 -> 0.33 ms, one protein pair of 383 residues 20 -> 12 us.  What is
// left is the longest segment's own chain of steps.
constexpr uint32_t kRecCol = 0xFFFFFu;  // column (pairs are below 2^20), state << 20, leave << 22
constexpr uint32_t kRecArrival = 0x3FFFFFu;
constexpr uint32_t kLeaveDiag = 0u << 22, kLeaveUp = 1u << 22, kLeaveStop = 2u << 22;
constexpr uint32_t kExitStop = 1u << 30, kExitBad = 1u << 31;  // exits: the path ends inside; the planes make no sense
constexpr int kSegRows = 64;  // fewest rows of a segment: paths meet within some tens of rows
constexpr int kWinSteps4 = 32, kWinLanes4 = 14, kWinSteps8 = 64, kWinLanes8 = 9, kWinWords = 576;
constexpr int kMaxSegs = 32;
static_assert(kWalkRecRows < ((222 << 10) / 4 - kMaxSegs * kWinWords), "shorter pairs' records fit");
constexpr size_t kWalkSmem = size_t(222) << 10;  // dynamic shared memory of a block, at most

struct SegWalk {
  uint32_t exit;  // arrival in row `lo`, or kExitStop and the column where the path ends
  int floor;      // last row walked
  bool met;       // met the recorded path: exit and floor are those it had
};

// Walks rows i = hi .. lo + 1 from (hi, j, state); writes their records.
// floor: the last row of the path recorded before (hi + 1: none).
template <class Plane>
__device__ __forceinline__ SegWalk walk_segment(Plane &pl, uint32_t *rec, int hi, int lo, int j, int state, bool local,
                                                int floor, int lane) {
  int i = hi;
  uint32_t arrival = uint32_t(j) | uint32_t(state) << 20;
  pl.set_row(i);
  // Leaves p rows, each `left` columns further left, arriving in the next with
  // `st` (the state's bits).  True when one of the rows it arrives in was arrived
  // in like that before.
  auto advance = [&](int p, int left, uint32_t st, uint32_t leave) {
    const int rk = i - 1 - lane;  // arrived in from row i - lane
    const bool same = lane < p && rk >= max(floor, lo + 1) &&
                      (rec[rk] & kRecArrival) == (uint32_t(j - left * (lane + 1)) | st);
    const uint32_t hit = __ballot_sync(0xffffffffu, same);
    const int q = hit ? __ffs(hit) : p;
    if (lane < q) rec[i - lane] = (lane == 0 ? arrival : uint32_t(j - left * lane) | st) | leave;
    i -= p;
    j -= left * p;
    arrival = uint32_t(j) | st;
    if (i > lo) pl.set_row(i);
    return hit != 0u;
  };
  for (;;) {
    if (state == 0) {
      if (j == 0) {
        if (local) {
          if (lane == 0) rec[i] = arrival | kLeaveStop;
          return {kExitStop, i, false};
        }
        // Global, left column: up to row 0.
        for (int k = i - lane; k > lo; k -= 32) rec[k] = (k == i ? arrival : 0u) | kLeaveUp;
        return {0u, lo + 1, false};
      }
      const int hd = pl.dir(j);
      if (hd == kDirDiag) {
        // A run of diagonal moves at once: lane k leaves row i - k.
        const uint32_t dm = pl.diag_mask(i, j);
        const int p = min(dm == 0xffffffffu ? 32 : __ffs(~dm) - 1, i - lo);
        if (advance(p, 1, 0u, kLeaveDiag)) return {0u, 0, true};
        if (i == lo) break;
      } else if (hd == kDirStop) {
        if (lane == 0) rec[i] = arrival | kLeaveStop;
        return {kExitStop | (local ? 0u : kExitBad) | uint32_t(j), i, false};
      } else {
        state = hd;
      }
    } else {
      // E and F runs end inside the matrix; if the planes say otherwise, stop.
      // The cells that extend the gap at once, the one that opened it by itself
      // (128 x 20,000, one long gap: 3.79 ms a call cell by cell, 1.89 like this).
      if (j <= 0) return {kExitBad | kExitStop, i, false};
      (void)pl.nib(j);
      const uint32_t gm = state == 1 ? pl.template gap_mask<true>(i, j) : pl.template gap_mask<false>(i, j);
      const int p = gm == 0xffffffffu ? 32 : __ffs(~gm) - 1;
      if (state == 1) {
        j -= max(p, 1);
        if (p == 0) state = 0;
      } else {
        if (p == 0) state = 0;
        if (advance(min(max(p, 1), i - lo), 0, uint32_t(state) << 20, kLeaveUp)) return {0u, 0, true};
        if (i == lo) break;
      }
    }
  }
  return {arrival, lo + 1, false};
}

template <int R>
__global__ void __launch_bounds__(kMaxSegs * 32) walk_block_kernel(const WalkArgs A) {
  extern __shared__ __align__(16) uint32_t s_dyn[];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ uint32_t s_entry[kMaxSegs], s_exit[kMaxSegs];
  __shared__ int s_floor[kMaxSegs];
  __shared__ int s_cols[kMaxSegs], s_ident[kMaxSegs];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int q = blockIdx.x;
  const int p = A.tasks[q];
  ResultDev &res = A.res[p];
  if (res.status != TSQ_OK) return;
  const PairDev pr = A.pairs[p];
  const int m = pr.a_len, n = pr.b_len;
  const bool local = A.local != 0, emit = A.emit != 0;
  if (local && res.score <= 0) {
    if (threadIdx.x == 0) {
      res.a_begin = res.a_end = res.b_begin = res.b_end = 0;
      res.n_ident = res.n_cols = 0;
    }
    return;
  }
  const int ie = local ? res.a_end : m, je = local ? res.b_end : n;
  // Records of rows 0..ie: shared memory where they fit.
  uint32_t *rec = ie < A.rec_words ? s_dyn + warps * kWinWords
                                   : reinterpret_cast<uint32_t *>(A.rec_rows + A.rec_off[q]);
  using Plane = WarpPlane<R, R == 4 ? kWinSteps4 : kWinSteps8, R == 4 ? kWinLanes4 : kWinLanes8>;
  static_assert(Plane::kWords <= kWinWords, "windows fit");
  const int G = A.shape_G[p];
  Plane pl{reinterpret_cast<const uint32_t *>(A.planes + A.plane_off[p]), s_dyn + w * kWinWords,
           Plane::band_words(n, G), 31 - __clz(G), lane, local ? 3u : 1u};
  const int segs = max(1, min(warps, ie / kSegRows));
  auto row_of = [&](int k) { return int(int64_t(ie) * k / segs); };
  const int lo = w < segs ? row_of(w) : 0, hi = w < segs ? row_of(w + 1) : 0;
  const bool works = w < segs && ie > 0;

  // ---- the path ----
  auto store = [&](uint32_t entry, const SegWalk &r) {
    if (lane == 0) {
      s_entry[w] = entry;
      if (!r.met) {
        s_exit[w] = r.exit;
        s_floor[w] = r.floor;
      }
    }
  };
  if (works) {
    int j = je;
    if (w < segs - 1) j = max(local ? je - (ie - hi) : int(int64_t(je) * hi / ie), min(je, 1));
    store(uint32_t(j), walk_segment(pl, rec, hi, lo, j, 0, local, hi + 1, lane));
  }
  __syncthreads();
  for (int round = 0; round < segs; ++round) {
    const uint32_t entry = works && w < segs - 1 ? s_exit[w + 1] : kExitStop;
    const bool again = !(entry & kExitStop) && entry != s_entry[w];
    if (!__syncthreads_or(again)) break;
    if (again)
      store(entry, walk_segment(pl, rec, hi, lo, int(entry & kRecCol), int(entry >> 20) & 3, local, s_floor[w], lane));
    __syncthreads();
  }
  // The path ends at (bi, bj), in segment `last`.
  int last = segs - 1, bi = 0, bj = 0;
  if (ie > 0) {
    while (last > 0 && !(s_exit[last] & kExitStop)) --last;
    const uint32_t exit = s_exit[last];
    if (exit & kExitBad) {  // cannot happen with valid planes
      if (threadIdx.x == 0) res.status = TSQ_E_CUDA;
      return;
    }
    if (exit & kExitStop) {
      bi = s_floor[last];
      bj = int(exit & kRecCol);
    } else {
      if (local) bj = int(exit & kRecCol);
      if (threadIdx.x == 0) rec[0] = (exit & kRecCol) | kLeaveStop;
    }
  } else if (threadIdx.x == 0) {
    rec[0] = uint32_t(je) | kLeaveStop;
  }
  __syncthreads();

  // ---- the columns: rows ie down to bi, an even share per warp ----
  const int total = ie - bi + 1;
  const int t0 = int(int64_t(total) * w / warps), t1 = int(int64_t(total) * (w + 1) / warps);
  // Columns of b against gaps in row i, the column it leaves by (next), how.
  struct Row {
    int run, next;
    uint32_t leave;
  };
  auto row = [&](int i) {
    const uint32_t v = rec[i];
    Row r;
    r.leave = v & (kLeaveUp | kLeaveStop);
    r.next = r.leave == kLeaveStop ? bj : int(rec[i - 1] & kRecCol);
    r.run = int(v & kRecCol) - r.next - (r.leave == kLeaveDiag ? 1 : 0);
    return r;
  };
  int cols = 0;
  for (int t = t0 + lane; t < t1; t += 32) {
    const Row r = row(ie - t);
    cols += r.run + (r.leave != kLeaveStop ? 1 : 0);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cols += __shfl_xor_sync(0xffffffffu, cols, o);
  if (lane == 0) s_cols[w] = cols;
  __syncthreads();
  int64_t off = 0;  // columns below this warp's rows
  int length = 0;
  for (int k = 0; k < warps; ++k) {
    if (k < w) off += s_cols[k];
    length += s_cols[k];
  }
  const int64_t cap = (int64_t)m + n;
  char *end_a = emit ? A.aln + A.aln_off[p] + cap - 1 : nullptr, *end_b = emit ? end_a + cap : nullptr;
  const uint8_t *sa = A.seqs + pr.a_off, *sb = A.seqs + pr.b_off;
  int ident = 0;
  for (int t = t0; t < t1; t += 32) {
    const int i = ie - t - lane;
    Row r{0, 0, kLeaveStop};
    if (t + lane < t1) r = row(i);
    const int c = r.run + (r.leave != kLeaveStop ? 1 : 0);
    int sum = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      sum += lane >= o ? v : 0;
    }
    const int64_t pos = off + sum - c;
    off += __shfl_sync(0xffffffffu, sum, 31);
    if (r.leave != kLeaveStop) {
      const uint8_t ca = sa[i - 1], cb = r.leave == kLeaveDiag ? sb[r.next] : uint8_t('-');
      ident += r.leave == kLeaveDiag && ca == cb;
      if (emit) {
        end_a[-(pos + r.run)] = char(ca);
        end_b[-(pos + r.run)] = char(cb);
      }
    }
    if (!emit) continue;
    // Gaps in a: short ones by their lane, long ones by the warp.
    const int top = r.next + r.run + (r.leave == kLeaveDiag ? 1 : 0);  // the arrival column
    if (r.run <= 32)
      for (int x = 0; x < r.run; ++x) {
        end_a[-(pos + x)] = '-';
        end_b[-(pos + x)] = char(sb[top - 1 - x]);
      }
    for (uint32_t far = __ballot_sync(0xffffffffu, r.run > 32); far; far &= far - 1) {
      const int k = __ffs(far) - 1;
      const int run = __shfl_sync(0xffffffffu, r.run, k), from = __shfl_sync(0xffffffffu, top, k);
      const int64_t at = __shfl_sync(0xffffffffu, pos, k);
      for (int x = lane; x < run; x += 32) {
        end_a[-(at + x)] = '-';
        end_b[-(at + x)] = char(sb[from - 1 - x]);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ident += __shfl_xor_sync(0xffffffffu, ident, o);
  if (lane == 0) s_ident[w] = ident;
  __syncthreads();
  if (threadIdx.x != 0) return;
  ident = 0;
  for (int k = 0; k < warps; ++k) ident += s_ident[k];
  if (emit || !local) {
    res.a_begin = bi;
    res.b_begin = bj;
  }
  if (!local) {
    res.a_end = m;
    res.b_end = n;
  }
  res.n_cols = length;
  res.n_ident = ident;
}

// ASCII -> letter codes, and (when clut is set) -> score classes for the
// int16x2 fill, through shared-memory tables.
__global__ void encode_kernel(const uint8_t *__restrict__ seqs, int64_t len, const uint8_t *__restrict__ lut,
                              uint8_t *__restrict__ codes, const uint8_t *__restrict__ clut,
                              uint8_t *__restrict__ ccodes, uint4 *__restrict__ zero, int64_t nzero) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ uint8_t s_lut[256], s_clut[256];
  s_lut[threadIdx.x] = lut[threadIdx.x];
  s_clut[threadIdx.x] = clut ? clut[threadIdx.x] : uint8_t(0);
  __syncthreads();
  // 16 residues per thread per iteration through 128-bit loads where the
  // buffer allows it; the tail goes byte by byte.
  const int64_t nvec = len / 16;
  const uint4 *src = reinterpret_cast<const uint4 *>(seqs);
  uint4 *dst = reinterpret_cast<uint4 *>(codes);
  uint4 *cdst = reinterpret_cast<uint4 *>(ccodes);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nzero; v += stride)
    zero[v] = make_uint4(0u, 0u, 0u, 0u);
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += stride) {
    const uint4 w0 = src[v];
    uint4 w = w0, c = w0;
    uint32_t *x = reinterpret_cast<uint32_t *>(&w);
    uint32_t *y = reinterpret_cast<uint32_t *>(&c);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t u = x[q];
      x[q] = uint32_t(s_lut[u & 0xFF]) | (uint32_t(s_lut[(u >> 8) & 0xFF]) << 8) |
             (uint32_t(s_lut[(u >> 16) & 0xFF]) << 16) | (uint32_t(s_lut[u >> 24]) << 24);
      y[q] = uint32_t(s_clut[u & 0xFF]) | (uint32_t(s_clut[(u >> 8) & 0xFF]) << 8) |
             (uint32_t(s_clut[(u >> 16) & 0xFF]) << 16) | (uint32_t(s_clut[u >> 24]) << 24);
    }
    dst[v] = w;
    if (ccodes) cdst[v] = c;
  }
  for (int64_t k = nvec * 16 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < len; k += stride) {
    codes[k] = s_lut[seqs[k]];
    if (ccodes) ccodes[k] = s_clut[seqs[k]];
  }
}

}  // namespace

cudaError_t launch_walk(const WalkArgs &a, cudaStream_t st) {
  if (a.n_tasks <= 0) return cudaSuccess;
  const int blocks = (a.n_tasks + kWarpWalkWarps - 1) / kWarpWalkWarps;
  if (a.n_tasks <= kWideWalks)
    walk_warp_kernel<true><<<blocks, kWarpWalkWarps * 32, 0, st>>>(a);
  else
    walk_warp_kernel<false><<<blocks, kWarpWalkWarps * 32, 0, st>>>(a);
  return cudaGetLastError();
}

// Warps of the many-warps walk: a segment each of at least kSegRows rows, and
// over all pairs about two warps for every place on the GPU.
cudaError_t launch_walk_block(const WalkArgs &args, int R, int32_t max_rows, cudaStream_t st, bool early) {
  if (args.n_tasks <= 0) return cudaSuccess;
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int share = std::max(4, sms * kMaxSegs * 2 / args.n_tasks);
  const int warps = std::max(1, std::min({kMaxSegs, share, max_rows / kSegRows}));
  const size_t windows = size_t(warps) * kWinWords * 4;
  WalkArgs a = args;
  a.rec_words = int32_t(std::min<size_t>((kWalkSmem - windows) / 4, size_t(max_rows) + 1));
  const size_t smem = windows + size_t(a.rec_words) * 4;
  auto kernel = R == 4 ? walk_block_kernel<4> : walk_block_kernel<8>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kWalkSmem));
  if (e != cudaSuccess) return e;
  return launch_maybe_early(kernel, dim3(a.n_tasks), warps * 32, smem, st, early, a);
}

cudaError_t launch_encode(const uint8_t *seqs, int64_t len, const uint8_t *lut_dev, uint8_t *codes,
                          const uint8_t *clut_dev, uint8_t *ccodes, cudaStream_t st, void *zero, int64_t zero_bytes) {
  if (len <= 0 && zero_bytes <= 0) return cudaSuccess;
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t work = std::max(len + 15, zero_bytes) / 16;
  int blocks = int(std::min<int64_t>((work + 255) / 256, (int64_t)sms * 8));
  if (blocks < 1) blocks = 1;
  encode_kernel<<<blocks, 256, 0, st>>>(seqs, len, lut_dev, codes, clut_dev, ccodes, static_cast<uint4 *>(zero),
                                      zero_bytes / 16);
  return cudaGetLastError();
}

}  // namespace tsq
