// pair.cpp -- the plain form's one-pair path (tsq_align_pair).
//
// A lone pair needs none of the batch planner's passes (per-pair checks
// over worker threads, lane types, radix sorts, warp-task lists) nor its
// dozen separate uploads and three host synchronisations.  This path packs
// everything the kernels read -- the pair record, its task entries, the
// zeroed work counter, the code tables, the score matrices and the
// residues -- into one page-locked block and sends it with one copy; runs
// the encoder, the fill and, for alignments, the walker; and brings the
// result record and the aligned rows back with one copy: one host
// synchronisation per call.
//
// The fill is a strip fill, in the kind of strips StripLoad estimates to
// finish first: the whole GPU is idle but for this pair, and one warp is the
// slowest way to sweep it (383 x 383 residues with traceback: 101 us on one
// int16x2 warp, 55 us in strips; 3,001 x 3,001 local 4,310 and 470 us).
// Identity output takes the traceback fill as well and walks it without
// writing rows; it falls back to the batch engine, which keeps no planes,
// when there is no memory for them.
// Scores, coordinates and rows are the same in every lane type.  Calls
// that force the checked int16x2 lane (TSQ_LANE_I16) and pairs outside
// pair_limits go to the batch engine (kPairNotTaken), which owns those
// cases and their error codes.
//
// The entry point this serves is the plain aligner call of the editor's
// "Align selection" (tweakseq/UI/SeqEditMainWin.cpp:1616-1663), one pair
// at a time.
#include <algorithm>
#include <cstring>

#include "engine.h"
#include "trace.h"

namespace tsq {

namespace {

#define PAIR_TRY(expr)                                  \
  do {                                                  \
    const cudaError_t e_ = (expr);                      \
    if (e_ != cudaSuccess) return cuda_status(e_);      \
  } while (0)

constexpr int64_t align256(int64_t x) { return (x + 255) & ~int64_t(255); }

// The upload block (byte offsets).  The device keeps a copy of it at the
// start of PairPath::dev; the kernels read every table there.
constexpr size_t kOffPair = 0;        // PairDev: a at kOffSeqs, b right after it
constexpr size_t kOffTask = 32;       // int32 pair id 0
constexpr size_t kOffCounter = 36;    // int32 work-queue head, zero
constexpr size_t kOffShapeG = 56;     // int32 G of the traceback planes
constexpr size_t kOffShapeR = 60;     // int32 R of the traceback planes
constexpr size_t kOffPlaneOff = 64;   // int64 0
constexpr size_t kOffAlnOff = 72;     // int64 0
constexpr size_t kOffRowOff = 80;     // int64 0: the strips' hand-over row
constexpr size_t kOffCtl = 96;        // StripCtl, zero
constexpr size_t kOffLut = 128;       // letter codes by byte
constexpr size_t kOffClut = 384;      // score classes by byte
constexpr size_t kOffMatrix = 640;    // 26 x 26 scores
constexpr size_t kOffCmatrix = 1344;  // nclasses x nclasses class scores
constexpr size_t kOffSeqs = 2048;     // residues of a, then b, then kPad zero bytes
// The fill's staging reads up to 64 bytes past a sequence; the zero bytes
// there encode to class 0 (and an invalid letter code, which no check
// reads past a sequence's end).
constexpr int64_t kPad = 128;
static_assert(kOffCtl + sizeof(StripCtl) <= kOffLut, "record overlaps the tables");
static_assert(kOffCmatrix + kLetters * kLetters <= kOffSeqs, "tables overlap the residues");
static_assert(sizeof(PairDev) <= kOffTask && sizeof(ResultDev) == 32, "record sizes");

}  // namespace

PairLayout pair_layout(int32_t la, int32_t lb, StripKind kind, int out_mode) {
  const bool walk = out_mode != kOutScore, emit = out_mode == kOutTrace;
  const int64_t len = int64_t(la) + lb;
  PairLayout l;
  l.up_bytes = int64_t(kOffSeqs) + len + kPad;
  l.codes = align256(l.up_bytes);
  l.ccodes = l.codes + align256(len + kPad);
  l.res = l.ccodes + align256(len + kPad);
  l.down_bytes = int64_t(sizeof(ResultDev)) + (emit ? 2 * len : 0);
  l.row = l.res + align256(l.down_bytes);
  l.row_bytes = 8 * strip_row_entries(la, lb, strip_rows(kind), walk);
  l.planes = l.row + align256(l.row_bytes);
  l.total = l.planes + std::max<int64_t>(walk ? plane_bytes(la, lb, strip_shape(kind)) : 0, 16);
  return l;
}

void PairPath::reset() {
  if (stream) cudaStreamSynchronize(stream);
  dev.release();
  up.release();
  down.release();
  if (stream) cudaStreamDestroy(stream);
  stream = nullptr;
  device = -1;
}

int pair_align(PairPath *pp, const uint8_t *a, int32_t la, const uint8_t *b, int32_t lb, const tsq_params *p,
               tsq_result *out) {
  if (!pp || !p || !out) return kPairNotTaken;
  if (check_params(p) != TSQ_OK || p->lane == TSQ_LANE_I16) return kPairNotTaken;
  Scheme sc;
  if (build_scheme(p, &sc) != TSQ_OK) return kPairNotTaken;
  const int out_mode = out_mode_of(p);
  const bool local = p->mode == TSQ_LOCAL;
  if (pair_limits(p, sc, out_mode, la, lb) != TSQ_OK) return kPairNotTaken;
  TraceRange tr("align pair (one-pair path)");

  int devno = 0;
  PAIR_TRY(cudaGetDevice(&devno));
  if (pp->device != devno) {
    pp->reset();
    PAIR_TRY(cudaStreamCreateWithFlags(&pp->stream, cudaStreamNonBlocking));
    PAIR_TRY(cudaDeviceGetAttribute(&pp->sms, cudaDevAttrMultiProcessorCount, devno));
    pp->device = devno;
  }
  cudaStream_t st = pp->stream;
  // Whatever this call returns, its copies have landed before the next call
  // rewrites the page-locked blocks.
  struct SyncOnExit {
    cudaStream_t st;
    ~SyncOnExit() { cudaStreamSynchronize(st); }
  } sync_on_exit{st};

  // ---- kind of strips ------------------------------------------------------
  const bool walk = out_mode != kOutScore, emit = out_mode == kOutTrace;
  const int fill_mode = walk ? kOutTrace : kOutScore;
  StripLoad load;
  load.add(la, lb);
  const StripKind kind = load.pick(
      fill_mode, pp->sms, p->lane == TSQ_LANE_AUTO && strip16_supported(sc, p->gap_open, p->gap_extend));
  const Shape shp = strip_shape(kind);
  const int n_units = std::max(1, (la + strip_rows(kind) - 1) / strip_rows(kind));
  const int blocks_avail = strip_blocks(kind, fill_mode, local, sc.nclasses);
  if (blocks_avail <= 0) return TSQ_E_CUDA;

  // ---- device block ----------------------------------------------------
  const int64_t len = int64_t(la) + lb;
  const PairLayout lay = pair_layout(la, lb, kind, out_mode);

  auto grow = [](size_t need, size_t cap) { return need <= cap ? need : need + need / 2; };
  // (A pair whose traceback planes do not fit in device memory fails here
  // with TSQ_E_NOMEM, as it does on the batch engine's one-pair plan.)
  cudaError_t e = pp->dev.ensure(grow(size_t(lay.total), pp->dev.cap), st);
  if (e == cudaErrorMemoryAllocation) {  // (without room to grow)
    cudaGetLastError();
    e = pp->dev.ensure(size_t(lay.total), st);
  }
  if (e != cudaSuccess) {
    if (e != cudaErrorMemoryAllocation || emit || !walk) return cuda_status(e);
    cudaGetLastError();
    return kPairNotTaken;
  }
  PAIR_TRY(pp->up.ensure(grow(size_t(lay.up_bytes), pp->up.cap)));
  PAIR_TRY(pp->down.ensure(grow(size_t(lay.down_bytes), pp->down.cap)));

  // ---- the upload block --------------------------------------------------
  uint8_t *h = pp->up.as<uint8_t>();
  std::memset(h, 0, kOffSeqs);
  const PairDev pd{0, la, la, lb};  // offsets into the residues
  std::memcpy(h + kOffPair, &pd, sizeof(pd));
  std::memcpy(h + kOffShapeG, &shp.G, sizeof(int32_t));
  std::memcpy(h + kOffShapeR, &shp.R, sizeof(int32_t));
  build_lut(sc, h + kOffLut);
  build_class_lut(sc, h + kOffClut);
  std::memcpy(h + kOffCmatrix, sc.cscore, size_t(sc.nclasses) * size_t(sc.nclasses));
  std::memcpy(h + kOffMatrix, sc.score, size_t(kLetters) * kLetters);
  if (la) std::memcpy(h + kOffSeqs, a, size_t(la));
  if (lb) std::memcpy(h + kOffSeqs + la, b, size_t(lb));
  std::memset(h + kOffSeqs + len, 0, size_t(kPad));

  uint8_t *d = pp->dev.as<uint8_t>();
  const uint8_t *seqs = d + kOffSeqs;
  uint8_t *codes = d + lay.codes;
  uint8_t *ccodes = d + lay.ccodes;
  ResultDev *res = reinterpret_cast<ResultDev *>(d + lay.res);
  PAIR_TRY(cudaMemcpyAsync(d, h, size_t(lay.up_bytes), cudaMemcpyHostToDevice, st));
  // (It also clears the hand-over row, and the launches after it start early: the
  // gaps between a short pair's launches are a tenth of its call.)
  PAIR_TRY(launch_encode(seqs, len + kPad, d + kOffLut, codes, d + kOffClut, ccodes, st, d + lay.row, lay.row_bytes));

  // ---- fill ----------------------------------------------------------------
  FillArgs fa{};
  fa.codes = codes;
  fa.pairs = reinterpret_cast<const PairDev *>(d + kOffPair);
  fa.tasks = reinterpret_cast<const int32_t *>(d + kOffTask);
  fa.wtasks = nullptr;  // one pair's strips in order
  fa.n_wtasks = n_units;
  fa.counter = reinterpret_cast<int32_t *>(d + kOffCounter);
  fa.matrix = reinterpret_cast<const int8_t *>(d + kOffMatrix);
  fa.gap_open = p->gap_open;
  fa.gap_extend = p->gap_extend;
  fa.res = res;
  fa.planes = d + lay.planes;
  fa.plane_off = reinterpret_cast<const int64_t *>(d + kOffPlaneOff);
  fa.max_score = sc.max_score;
  fa.ccodes = ccodes;
  fa.cmatrix = reinterpret_cast<const int8_t *>(d + kOffCmatrix);
  fa.nclasses = sc.nclasses;
  fa.strip_ctl = reinterpret_cast<StripCtl *>(d + kOffCtl);
  fa.strip_rows = reinterpret_cast<uint64_t *>(d + lay.row);
  fa.strip_row_off = reinterpret_cast<const int64_t *>(d + kOffRowOff);
  PAIR_TRY(launch_strip(kind, fill_mode, local, fa, std::min(blocks_avail, n_units), st, true));

  // ---- traceback ---------------------------------------------------------
  char *rows = reinterpret_cast<char *>(d + lay.res + sizeof(ResultDev));
  if (walk) {
    WalkArgs w{};
    w.seqs = seqs;
    w.codes = codes;
    w.pairs = fa.pairs;
    w.tasks = fa.tasks;
    w.n_tasks = 1;
    w.planes = fa.planes;
    w.plane_off = fa.plane_off;
    w.shape_G = reinterpret_cast<const int32_t *>(d + kOffShapeG);
    w.shape_R = reinterpret_cast<const int32_t *>(d + kOffShapeR);
    w.local = local ? 1 : 0;
    w.emit = emit ? 1 : 0;
    w.res = res;
    w.aln = rows;
    w.aln_off = reinterpret_cast<const int64_t *>(d + kOffAlnOff);
    w.rec_rows = fa.strip_rows;
    w.rec_off = fa.strip_row_off;
    PAIR_TRY(launch_walk_block(w, shp.R, la, st, true));
  }
  PAIR_TRY(cudaMemcpyAsync(pp->down.p, res, size_t(lay.down_bytes), cudaMemcpyDeviceToHost, st));
  PAIR_TRY(cudaStreamSynchronize(st));

  const ResultDev rd = *pp->down.as<ResultDev>();
  const char *hrows = pp->down.as<char>() + sizeof(ResultDev);
  const int rc = collect_one(rd, emit && rd.status == TSQ_OK ? hrows : nullptr, len, *out);
  if (rc) return rc;
  return rd.status;
}

}  // namespace tsq
