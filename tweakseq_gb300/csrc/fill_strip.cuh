// fill_strip.cuh -- pieces shared by the strip fills (fill_strip32.cuh,
// fill_strip16.cuh): one pair spread over many warps of the whole GPU.
//
// The rows of a pair are cut into strips; one warp fills one strip, left to
// right, its lanes one column apart.  A strip's bottom row is the top row of
// the next, and consecutive strips run at the same time, each a few dozen
// columns behind the one above: a pair of m rows keeps m / (rows per strip)
// warps busy, on as many SMs, instead of the warps of one CTA (a 20 kb pair
// with traceback ran 32.0 ms on one 16-warp CTA).
//
// Work.  A unit is one strip of one pair.  Warps claim units from one
// counter.  The list is ordered so that a pair's strips appear in order, so
// the strip that a warp waits for is finished or is held by a warp that is
// already running: no waiting cycle, whatever the number of resident warps.
// Across pairs the order is by the work that is left below a strip, most
// first, so that the longest pair is not the tail.
//
// Hand-over.  Each pair has one row of n 64-bit entries in global memory:
// H (30 bits: every score is within 2^28), H - F (20 bits, cut at open + 1: a
// larger difference opens the next F in any case) and a tag, one more than
// the number of the strip that wrote the entry (14 bits; 1,048,575 rows are
// 8,192 strips of 128).  Every strip of a pair has its own tag: strips that are far
// ahead in the list may already wait on an entry that is rewritten many times
// before their turn.  The
// tag travels with the data in one 64-bit store, so a reader needs no
// counter and no fence: it loads the entries of the next chunk of columns
// one chunk ahead and takes them when every tag is the one it wants.  The row
// is rewritten in place: strip s + 1 writes column j after reading it, and
// strip s is past j by then.  The rows are cleared before each run (tag 0 is
// never expected), so entries of an earlier run are not taken for new ones.
//
// Every wait is bounded (FillArgs::spin_limit polls).  A wait that runs out
// marks the pair TSQ_E_TIMEOUT; the strip then goes on without waiting, with
// the entries it has, and publishes as usual, so the kernel always ends.  It may
// overtake the strip above, which then writes over entries that the strip below
// has not read: that one runs its own limit out, and so may each further down, most
// of them at the same time (a strip waits for its limit once).  (Looking at the
// pair's mark in the poll loop would end them at once; it cost the fills 1 to 2 %.)
// Every index it uses stays inside its rings, the pair's row and the pair's planes.
#pragma once

#include <cstdint>

#include "fill_common.cuh"

namespace tsq {
namespace fill {

// Polls of a wait by default: about 0.7 s for the strip above, 35 s where a strip's
// turn is far off and it sleeps between them.
constexpr int kStripPolls = 1 << 20;

constexpr uint32_t kTagMask = 0x3FFFu;  // tags 1..16383
static_assert((kMaxPairLen + 127) / 128 - 1 <= int64_t(kTagMask), "a tag for every strip that hands down");

// Lets the next launch start (it waits for this one), and waits for the one ahead,
// where the launches allow it (launch_maybe_early).
__device__ __forceinline__ void strip_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t strip_tag(int strip) { return uint32_t(strip) + 1u; }

// (H, F) of a bottom-row cell as a tagged entry; dmax = open + 1.
__device__ __forceinline__ uint64_t strip_entry(int32_t h, int32_t f, int32_t dmax, uint32_t tag) {
  const uint32_t d = uint32_t(min(h - f, dmax)) & 0xFFFFFu;
  return (uint64_t(uint32_t(h) * 4u + (d >> 18)) << 32) | (d * (kTagMask + 1u) + tag);
}
__device__ __forceinline__ int32_t strip_h(uint64_t v) { return int32_t(uint32_t(v >> 32)) >> 2; }
__device__ __forceinline__ int32_t strip_f(uint64_t v) { return strip_h(v) - int32_t(uint32_t(v >> 14) & 0xFFFFFu); }

__device__ __forceinline__ uint64_t strip_load(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void strip_store(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The top row of one strip, read chunk by chunk (COLS columns, lane q column
// q of the chunk): `ahead` holds the entries of the next chunk, loaded one
// chunk early.
template <int COLS>
struct StripReader {
  const uint64_t *row;
  uint32_t tag;   // the tag of the strip above
  int n, lane, limit;
  bool gave_up;
  uint64_t ahead;
  __device__ uint64_t fetch(int chunk) const {
    const int col = COLS * chunk + lane;
    return lane < COLS && col < n ? strip_load(row + col) : uint64_t(tag);
  }
  // The entries of `chunk` (which `ahead` was loaded for), waiting until
  // they are there; then loads the next chunk's.
  __device__ uint64_t take(int chunk) {
    uint64_t v = ahead;
    for (int polls = 0; !__all_sync(0xffffffffu, (uint32_t(v) & kTagMask) == tag) && !gave_up;) {
      if (polls >= limit) {
        gave_up = true;
        break;
      }
      // The tag found says how many strips are still to write this entry.
      // All strips of a pair wait on the same few entries at first: each
      // sleeps about as long as the strips between take to get there (40
      // steps of some 50 ns each), or thousands of polls of one address would
      // hold the writer up.
      const uint32_t away = tag - __shfl_sync(0xffffffffu, uint32_t(v) & kTagMask, 0);
      const uint32_t ns = away <= 1u ? 0u : min(away, 64u) * 512u;
      ++polls;
      if (ns) __nanosleep(ns);
      v = fetch(chunk);
    }
    ahead = fetch(chunk + 1);
    return v;
  }
};

// A strip's end: its findings go to the pair's record, and the strip that
// finishes last (which strip that is does not matter) writes the result.
// flags: 1 an invalid residue, 2 a wait ran out.  key: the strip's local
// maximum as (score, -row, -column); last_h: H(m, n) on lane `owner` of the
// last strip (owner < 0 elsewhere).
__device__ __forceinline__ void strip_finish(const FillArgs &A, int q, int pid, int m, int n, int strips, int lane,
                                             int flags, uint64_t key, int owner, int32_t last_h, bool local,
                                             bool trace) {
  StripCtl *c = A.strip_ctl + q;
  if (lane == owner) c->last_h = last_h;
  if (lane == 0) {
    if (flags) atomicOr(&c->flags, flags);
    if (local && key) atomicMax(reinterpret_cast<unsigned long long *>(&c->key), static_cast<unsigned long long>(key));
  }
  __threadfence();
  __syncwarp();
  if (lane != 0) return;
  if (atomicAdd(&c->done, 1) != strips - 1) return;
  __threadfence();
  const int fl = *reinterpret_cast<volatile int32_t *>(&c->flags);
  const bool empty = m == 0 || n == 0;
  ResultDev &o = A.res[pid];
  o.status = (fl & 1) ? TSQ_E_INVALID_RESIDUE : ((fl & 2) ? TSQ_E_TIMEOUT : TSQ_OK);
  o.n_ident = o.n_cols = -1;
  if (local) {
    const uint64_t gkey = (fl & 1) ? 0u : *reinterpret_cast<volatile uint64_t *>(&c->key);
    const int32_t sc = int32_t(gkey >> 40);
    o.score = sc;
    o.a_end = sc > 0 ? int32_t(0xFFFFFu - uint32_t((gkey >> 20) & 0xFFFFFu)) : 0;
    o.b_end = sc > 0 ? int32_t(0xFFFFFu - uint32_t(gkey & 0xFFFFFu)) : 0;
    o.a_begin = o.b_begin = sc > 0 ? -1 : 0;
  } else {
    o.a_begin = 0;
    o.a_end = m;
    o.b_begin = 0;
    o.b_end = n;
    o.score = empty ? ((m + n == 0) ? 0 : -(A.gap_open + (m + n) * A.gap_extend))
                    : ((fl & 1) ? 0 : *reinterpret_cast<volatile int32_t *>(&c->last_h));
    if (trace && empty) {
      o.n_ident = 0;
      o.n_cols = m + n;
    }
  }
}

// True when any of the `len` letter codes at p is invalid; the warp's lanes
// read the 16-byte chunks covering the range.
__device__ __forceinline__ bool strip_has_bad(const uint8_t *p, int len, int lane) {
  if (len <= 0) return false;
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uintptr_t a0 = a & ~uintptr_t(15);
  const int head = int(a - a0);
  const int nch = (head + len + 15) >> 4;
  uint32_t any = 0;
#pragma unroll 4
  for (int c = lane; c < nch; c += 32) {
    const uint4 w = *reinterpret_cast<const uint4 *>(a0 + 16 * uintptr_t(c));
    const int s = head - 16 * c, e = head + len - 16 * c;  // bytes [s, e) of this chunk are in range
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int lo = min(max(s - 4 * q, 0), 4), hi = min(max(e - 4 * q, 0), 4);
      const uint32_t mlo = lo >= 4 ? 0u : (0xFFFFFFFFu << (8 * lo));
      const uint32_t mhi = hi >= 4 ? 0xFFFFFFFFu : ((1u << (8 * hi)) - 1u);
      any |= __vcmpgeu4(ww[q], 0x1A1A1A1Au) & mlo & mhi;
    }
  }
  return any != 0;
}

// Class codes of columns [32k, 32k + 32], lanes 0..2, into a ring of RING
// bytes whose first 16 bytes are mirrored past its end.
template <int RING>
__device__ __forceinline__ void strip_stage_codes(int k, int t, int n, const uint8_t *codes, int64_t boff,
                                                  uint8_t *ring) {
  const int c0 = kChunk * k;
  if (c0 >= n || t >= 3) return;
  const int64_t a = ((boff + c0) & ~int64_t(15)) + 16 * t;
  cp_async16(ring + (a & (RING - 1)), codes + a);
  if ((a & (RING - 1)) == 0) cp_async16(ring + RING, codes + a);
}

}  // namespace fill
}  // namespace tsq
