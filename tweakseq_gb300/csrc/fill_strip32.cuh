// fill_strip32.cuh -- strip fill in int32 lanes: strips of 128 rows, four
// rows per lane (score and traceback output, global or local).
//
// For pairs that are few or alone: the lanes of a warp are one column apart,
// so the sweep of an m x n pair is one wavefront, whatever m, and int32 needs
// no second band of rows (which would put 32 more columns between strips) and
// no range rules.  A warp with a scheduler to itself issues one instruction
// in about 2.3 cycles whatever is independent (two columns a step, to fill
// waits, only made the strips start further apart: 2.33 against 1.94 ms on
// 20,000 x 20,000, score), so what counts is the instructions of a step.  Per
// cell the score fill issues 7, the traceback fill 14: each of the four
// decisions is the sign of one difference (an IMAD by an opaque -1, FMA
// pipe), shifted into a word by one funnel shift.  Beside its cells a step
// issues about 17: the shuffles that join the lanes, the code, profile and
// top-row reads, and an eighth of the hand-over.  (Two rows per lane, twice
// the strips: 2.19 against 1.83 ms there, 2.69 against 2.68 with traceback.)
//
// Traceback planes: words of eight cells, two steps.  Band b (= strip) of 128
// rows, step s = column + lane: lane t at word
// (b * ceil((n + 31) / 2) + s / 2) * 32 + t, row r of step s in nibble
// 7 - (s % 2 * 4 + r), the nibble as in the other fills (bits 0-1 direction,
// bit 2 E opened, bit 3 F opened).
#pragma once

#include <algorithm>
#include <cstdint>

#include "fill_i16.cuh"
#include "fill_strip.cuh"

namespace tsq {
namespace fill {

constexpr int kStripRows32 = 128;
constexpr int kStripCols32 = 8;  // columns per hand-over chunk

__host__ __device__ constexpr size_t strip32_smem_bytes(int nclasses) {
  return size_t(kMatBytes16) + size_t(nclasses) * 32 * sizeof(uint32_t) + (kTopRing + 2) * sizeof(int2) +
         2 * kStripCols32 * sizeof(int2) + kCodeRing + kRingPad;
}

// acc * 2 + (d < 0).
__device__ __forceinline__ uint32_t push_sign(uint32_t acc, int32_t d) {
  return __funnelshift_l(uint32_t(d), acc, 1);
}

template <int OUT, bool LOCAL>
__global__ void __launch_bounds__(32) fill_strip32_kernel(const FillArgs A) {
  static_assert(OUT == kOutScore || OUT == kOutTrace, "score and traceback output");
  constexpr int R = 4, S = kStripRows32, C = kStripCols32, U = 8 / R;  // U: steps per plane word
  extern __shared__ __align__(16) uint8_t smem[];
  strip_begin();
  int8_t *s_mat = reinterpret_cast<int8_t *>(smem);
  uint32_t *s_prof = reinterpret_cast<uint32_t *>(smem + kMatBytes16);
  const int ncls = A.nclasses;
  int2 *top_ring = reinterpret_cast<int2 *>(smem + kMatBytes16 + size_t(ncls) * 32 * sizeof(uint32_t));
  int2 *out_ring = top_ring + kTopRing + 2;  // the bottom row's last 2 C columns
  uint8_t *code_ring = reinterpret_cast<uint8_t *>(out_ring + 2 * C);
  const int t = threadIdx.x;
  for (int k = t; k < kMatBytes16; k += 32) {
    const int x = k / kMatRow16, c = k % kMatRow16;
    s_mat[k] = (x < ncls && c < ncls) ? A.cmatrix[x * ncls + c] : int8_t(0);
  }
  // The code ring starts as class 0: positions that are read before their
  // columns are staged (the lane is out of range there) index the profile.
  for (int k = t; k < kCodeRing + kRingPad; k += 32) code_ring[k] = 0;
  __syncwarp();

  const int32_t go = A.gap_open, ge = A.gap_extend, oe = go + ge;
  const int32_t one = int32_t(A.one), minus_one = -one;
  const uint32_t *prof = s_prof + t;
  auto mad = [](int32_t a, int32_t b, int32_t c) { return int32_t(imad(uint32_t(a), uint32_t(b), uint32_t(c))); };

  for (;;) {
    int u = 0;
    if (t == 0) u = atomicAdd(A.counter, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= A.n_wtasks) break;
    const int2 unit = A.wtasks ? A.wtasks[u] : make_int2(0, u);
    const int q = unit.x, strip = unit.y;
    const int pid = A.tasks[q];
    const PairDev pr = A.pairs[pid];
    const int m = pr.a_len, n = pr.b_len;
    const int strips = max(1, (m + S - 1) / S);
    const int row0 = strip * S + t * R;  // rows row0+1 .. row0+R (1-based)
    int flags = 0;
    // Invalid residues: each strip checks its own rows, the first one also b.
    bool bad = strip_has_bad(A.codes + pr.a_off + strip * S, min(S, m - strip * S), t);
    if (strip == 0) bad |= strip_has_bad(A.codes + pr.b_off, n, t);
    if (__any_sync(0xffffffffu, bad)) flags = 1;
    uint64_t lkey = 0;
    int32_t last_h = 0;
    int owner = -1;

    if (m > 0 && n > 0) {
      // Profile: the scores of this lane's rows against each class.
      {
        const uint8_t *qa = A.ccodes + pr.a_off;
        int xa[R];
#pragma unroll
        for (int r = 0; r < R; ++r) xa[r] = kMatRow16 * (row0 + r < m ? int(qa[row0 + r]) : ncls);
#pragma unroll 1
        for (int cb = 0; cb < ncls; cb += 4) {
          uint32_t a[R], w[4];
#pragma unroll
          for (int r = 0; r < R; ++r) a[r] = *reinterpret_cast<const uint32_t *>(s_mat + xa[r] + cb);
          transpose4x4(a[0], a[1], a[2], a[3], w);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (cb + k < ncls) s_prof[(cb + k) * 32 + t] = w[k];
        }
      }
      uint64_t *row = A.strip_rows + A.strip_row_off[q];
      const uint32_t tag = strip_tag(strip);
      const bool hands_down = strip + 1 < strips;
      StripReader<C> rd{row, strip_tag(strip - 1), n, t, A.spin_limit > 0 ? A.spin_limit : kStripPolls, false, 0u};
      // Columns [C * chunk, C * chunk + C) of the top row go to the ring.
      auto take = [&](int chunk) {
        const int col = C * chunk + t;
        int2 v;
        if (strip > 0) {
          const uint64_t e = rd.take(chunk);
          v = make_int2(strip_h(e), strip_f(e));
        } else {
          v = make_int2(edge_h(col + 1, go, ge, LOCAL), kNegInf);
        }
        if (t < C) {
          top_ring[col & (kTopRing - 1)] = v;
          if ((col & (kTopRing - 1)) == 0) top_ring[kTopRing] = v;
        }
        __syncwarp();
      };
      // Hands chunk `chunk` of the bottom row down (its columns < n).
      auto give = [&](int chunk) {
        const int col = C * chunk + t;
        if (hands_down && t < C && unsigned(col) < unsigned(n)) {
          const int2 v = out_ring[(col - 1) & (2 * C - 1)];
          strip_store(row + col, strip_entry(v.x, v.y, go + 1, tag));
        }
      };
      cp_async_wait_all();
      __syncwarp();
      strip_stage_codes<kCodeRing>(0, t, n, A.ccodes, pr.b_off, code_ring);
      cp_async_commit();
      if (strip > 0) rd.ahead = rd.fetch(0);
      take(0);
      cp_async_wait_all();
      __syncwarp();
      strip_stage_codes<kCodeRing>(1, t, n, A.ccodes, pr.b_off, code_ring);
      cp_async_commit();

      int32_t H[R], E[R], T[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        H[r] = edge_h(row0 + r + 1, go, ge, LOCAL);
        T[r] = H[r] - oe;
        E[r] = kNegInf;
      }
      int32_t hdiag = edge_h(row0, go, ge, LOCAL);
      int32_t outH = 0, outF = kNegInf;
      // Local: each row's best score and the step of its first column.
      int32_t best[R], bstep[R];
#pragma unroll
      for (int r = 0; r < R; ++r) best[r] = bstep[r] = 0;
      (void)best, (void)bstep;
      uint32_t *plane = nullptr;
      if constexpr (OUT == kOutTrace)
        plane = reinterpret_cast<uint32_t *>(A.planes + A.plane_off[pid]) +
                int64_t(strip) * ((n + 31 + U - 1) / U) * 32 + t;
      uint32_t acc = 0u, stop = 0u;  // traceback: the decisions of the word's steps so far
      (void)plane, (void)acc, (void)stop;

      uint32_t pw[2];
      int2 tv[2];
      pw[0] = prof[int(code_ring[(pr.b_off - t) & (kCodeRing - 1)]) * 32];
      tv[0] = top_ring[0];
      const int steps_pad = (n + 31 + C + 7) & ~7;  // the last chunk is handed down within them
      const int i0 = min(32, steps_pad), i1 = max(i0, n & ~7);
      const int c0 = int(pr.b_off & (kCodeRing - 1)) - t + 1 + kCodeRing;  // code of column j + 1, positive

      auto step = [&](const int s, auto k_tag, auto interior_tag, const uint8_t *code, const int2 *topp,
                      int2 *outp) {
        constexpr int k = decltype(k_tag)::value;
        constexpr int cur = k & 1, nxt = cur ^ 1;
        constexpr bool INTERIOR = decltype(interior_tag)::value;
        const int32_t rH = __shfl_up_sync(0xffffffffu, outH, 1);
        const int32_t rF = __shfl_up_sync(0xffffffffu, outF, 1);
        const uint32_t w = pw[cur];
        pw[nxt] = prof[int(code[k]) * 32];
        const int32_t upH = t == 0 ? tv[cur].x : rH;
        const int32_t upF = t == 0 ? tv[cur].y : rF;
        tv[nxt] = topp[k];
        if (INTERIOR || unsigned(s - t) < unsigned(n)) {
          int32_t d = hdiag;
          hdiag = upH;
          int32_t xo = mad(upH, one, -oe);
          int32_t fv = upF;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int32_t sc = sbyte_dyn(w, r);
            const int32_t e = __viaddmax_s32(E[r], -ge, T[r]);
            const int32_t f = __viaddmax_s32(fv, -ge, xo);
            int32_t x = 0, h;
            if constexpr (OUT == kOutScore) {
              x = __viaddmax_s32(d, sc, e);
              h = LOCAL ? __vimax3_s32(x, f, 0) : max(x, f);
            } else {
              const int32_t dd = mad(sc, one, d);
              x = LOCAL ? max(dd, e) : 0;
              h = LOCAL ? __vimax3_s32(x, f, 0) : __vimax3_s32(dd, e, f);
              acc = push_sign(acc, mad(f, minus_one, xo));    // F extended
              acc = push_sign(acc, mad(e, minus_one, T[r]));  // E extended
              if constexpr (LOCAL) {
                acc = push_sign(acc, mad(h, minus_one, x));   // H not from X
                acc = push_sign(acc, mad(x, minus_one, dd));  // X from E
              } else {
                acc = push_sign(acc, mad(h, minus_one, e));   // H above E
                acc = push_sign(acc, mad(h, minus_one, dd));  // H not the diagonal's
              }
              if constexpr (LOCAL) stop |= uint32_t((h - 1) >> 31) & (3u << (4 * (7 - ((k % U) * R + r))));
            }
            T[r] = mad(h, one, -oe);
            // (Score: from X, a shorter chain through the rows: one pair of 20 kb
            // 1.86 ms, from H 2.05.)
            xo = OUT == kOutTrace ? T[r] : LOCAL ? __viaddmax_s32(x, -oe, -oe) : mad(x, one, -oe);
            E[r] = e;
            d = H[r];
            H[r] = h;
            fv = f;
            if constexpr (LOCAL) {
              const bool more = h > best[r];  // strictly: the first column of a maximum is kept
              best[r] = max(best[r], h);
              bstep[r] = more ? s : bstep[r];
            }
          }
          outH = H[R - 1];
          outF = fv;
        } else if (OUT == kOutTrace) {
          acc <<= 4 * R;
        }
        if (t == 31) outp[k] = make_int2(outH, outF);
        if constexpr (OUT == kOutTrace && k % U == U - 1) {
          // Local: E only where F does not win.  The opened bits are the
          // complements of the extended ones.
          uint32_t word = (LOCAL ? acc & ~((acc >> 1) & 0x11111111u) : acc) ^ 0xCCCCCCCCu;
          if constexpr (LOCAL) {
            word |= stop;
            stop = 0u;
          }
          if (INTERIOR || (s >= t && s - (U - 1) < t + n)) plane[int64_t(s / U) * 32] = word;
        }
      };
      int s0 = 0;
      // Units of eight steps.  Lane 31 puts column s - 31 of the bottom row at
      // place s mod 16, so chunk c is complete after step 8 (c + 4) + 6, and
      // goes down before a unit's last step.
      auto unit8 = [&](auto interior_tag) {
        const uint8_t *code = code_ring + ((c0 + s0) & (kCodeRing - 1));
        const int2 *topp = top_ring + ((s0 & (kTopRing - 1)) + 1);
        int2 *outp = out_ring + (s0 & (2 * C - 1));
        step(s0, IntTag<0>{}, interior_tag, code, topp, outp);
        step(s0 + 1, IntTag<1>{}, interior_tag, code, topp, outp);
        step(s0 + 2, IntTag<2>{}, interior_tag, code, topp, outp);
        step(s0 + 3, IntTag<3>{}, interior_tag, code, topp, outp);
        step(s0 + 4, IntTag<4>{}, interior_tag, code, topp, outp);
        step(s0 + 5, IntTag<5>{}, interior_tag, code, topp, outp);
        step(s0 + 6, IntTag<6>{}, interior_tag, code, topp, outp);
        take(s0 / C + 1);
        if (((s0 + 8) & (kChunk - 1)) == 0) {
          cp_async_wait_all();
          __syncwarp();
          strip_stage_codes<kCodeRing>((s0 + 8) / kChunk + 1, t, n, A.ccodes, pr.b_off, code_ring);
          cp_async_commit();
        }
        give(s0 / C - 4);
        step(s0 + 7, IntTag<7>{}, interior_tag, code, topp, outp);
        s0 += 8;
      };
#pragma unroll 1
      while (s0 < i0) unit8(BoolTag<false>{});
#pragma unroll 1
      while (s0 < i1) unit8(BoolTag<true>{});
#pragma unroll 1
      while (s0 < steps_pad) unit8(BoolTag<false>{});
      cp_async_wait_all();
      __syncwarp();
      if (rd.gave_up) flags |= 2;
      if constexpr (LOCAL) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (row0 + r < m && best[r] > 0) {
            const uint64_t key = (uint64_t(uint32_t(best[r])) << 40) |
                                 (uint64_t(0xFFFFFu - uint32_t(row0 + r + 1)) << 20) |
                                 uint64_t(0xFFFFFu - uint32_t(bstep[r] - t + 1));
            lkey = key > lkey ? key : lkey;
          }
        }
        lkey = group_max<32>(lkey);
      } else if (!hands_down) {
        const int lr = m - 1 - strip * S;  // row m within this strip
        owner = lr / R;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r == lr % R) last_h = H[r];
      }
    }
    strip_finish(A, q, pid, m, n, strips, t, flags, lkey, owner, last_h, LOCAL, OUT == kOutTrace);
    __syncwarp();
  }
}

}  // namespace fill
}  // namespace tsq
