// The one-pair path's device block: its parts hold what the kernels write and
// do not overlap.  Host code only.
#include <cstdio>

#include "engine.h"

using namespace tsq;

static int check(int32_t la, int32_t lb, StripKind kind, int out_mode) {
  const PairLayout l = pair_layout(la, lb, kind, out_mode);
  const bool walk = out_mode != kOutScore;
  const int64_t len = int64_t(la) + lb;
  // The walk's records, one 32-bit word for each of rows 0 to la, where they may
  // leave shared memory; the strips' hand-over entries, one for each column.
  const int64_t records = walk && la >= kWalkRecRows ? 4 * (int64_t(la) + 1) : 0;
  const int64_t entries = la > strip_rows(kind) ? 8 * int64_t(lb) : 0;
  const int64_t planes = walk ? plane_bytes(la, lb, strip_shape(kind)) : 0;
  const bool ok = l.up_bytes >= len && l.codes >= l.up_bytes && l.ccodes >= l.codes + len && l.res >= l.ccodes + len &&
                  l.down_bytes >= int64_t(sizeof(ResultDev)) + (out_mode == kOutTrace ? 2 * len : 0) &&
                  l.row >= l.res + l.down_bytes && l.row_bytes >= records && l.row_bytes >= entries &&
                  l.row_bytes % 16 == 0 && l.planes >= l.row + l.row_bytes && l.total >= l.planes + planes &&
                  l.codes % 16 == 0 && l.ccodes % 16 == 0 && l.res % 16 == 0 && l.row % 16 == 0 && l.planes % 16 == 0;
  if (!ok) {
    std::printf("la %d lb %d strips of %d rows output %d: row of %lld bytes, %lld before the planes; records %lld, "
                "entries %lld\n", la, lb, strip_rows(kind), out_mode, (long long)l.row_bytes, (long long)(l.planes - l.row),
                (long long)records, (long long)entries);
    return 1;
  }
  return 0;
}

int main() {
  int bad = 0;
  for (StripKind kind : {kStrip32, kStrip16})
    for (int out_mode : {kOutScore, kOutIdent, kOutTrace})
      for (int32_t lb : {0, 1, 15, 16, 17, 297, 301, 700, 10000, 19200, 25600, 65535}) {
        for (int32_t la : {0, 1, 127, 128, 129, 511, 512, 513, 32767, 1048575}) bad += check(la, lb, kind, out_mode);
        for (int32_t la = 32768; la < 33100; ++la) bad += check(la, lb, kind, out_mode);
        for (int32_t la = 38390; la < 38530; ++la) bad += check(la, lb, kind, out_mode);
        for (int32_t la : {39999, 40000, 40001, 51200, 524288, 1048512}) bad += check(la, lb, kind, out_mode);
      }
  if (bad) return 1;
  std::puts("layout ok");
  return 0;
}
