// tsq_internal.h -- shared declarations of the GB300 alignment library.
//
// Device data layout (all in HBM, one allocation pool per context):
//   codes      uint8 per residue: 'A'..'Z' -> 0..25 when the scheme accepts
//              the letter, kBadCode otherwise (converted once per batch).
//   ccodes     score batches: uint8 score class per residue, 0 for bytes
//              the scheme rejects (their codes entry marks them), and 128
//              bytes of class 0 past the residues: every entry indexes the
//              int16x2 fill's profile.
//   pairs      PairDev per pair (offsets into codes, lengths).
//   tasks      int32 pair ids of one launch, sorted so that the groups of a
//              warp get pairs of nearly the same shape.
//   results    ResultDev per pair.
//   boundary   per group slot, two rows of (H, F) of max_n + 1 columns: the
//              bottom row of one band of rows is the top row of the next.
//   planes     traceback nibbles (TB mode), diagonal-major per band so the
//              lanes of a group store one contiguous run per step.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstddef>

#include <cuda_runtime.h>

#include "../../include/tweakseq_gb300.h"

namespace tsq {

constexpr uint8_t kBadCode = 0xFF;
constexpr int kLetters = 26;
constexpr int32_t kNegInf = -(1 << 29);  // "minus infinity" for int32 E/F

// Longest sequence the int32 kernels take: coordinates travel in 20 bits.
constexpr int64_t kMaxPairLen = (1 << 20) - 1;

// Output modes of the fill kernels.
enum : int { kOutScore = 0, kOutIdent = 1, kOutTrace = 2 };
// Traceback nibble: bits 0-1 H source, bit 2 E opened, bit 3 F opened.
enum : int { kDirDiag = 0, kDirE = 1, kDirF = 2, kDirStop = 3 };
// The two low bits of a cell in the traceback planes.  Local: one of the above.
// Global: bit 0 H is not the diagonal's, bit 1 H is above E, so 0 and 2 stand for
// the diagonal, 1 for E and 3 for F (a bit less to work out per cell).
constexpr int kDirFGlobal = 3;

struct Scheme {
  int8_t score[kLetters][kLetters];
  uint8_t valid[kLetters];
  int32_t max_score, min_score;
  bool symmetric;
  // Score classes: valid letters with the same row and column of scores
  // (BLOSUM62: J, O, U and X) share a class; the int16x2 fills index their
  // profile by class, which keeps the profile small.  For identity output
  // every valid letter is its own class (identical = same class).
  int32_t nclasses;
  uint8_t cls[kLetters];               // class of each letter, kBadCode if invalid
  int8_t cscore[kLetters * kLetters];  // nclasses x nclasses class scores
};

struct PairDev {
  int64_t a_off, b_off;
  int32_t a_len, b_len;
};

struct ResultDev {
  int32_t score;
  int32_t a_begin, a_end, b_begin, b_end;
  int32_t n_ident, n_cols;
  int32_t status;
};

// Kernel shape of the group-striped fill: G lanes per pair, R rows per lane,
// int32 or int16x2 values.
struct Shape {
  int G, R, i16;
};

// What the strips of one pair leave for the one that finishes last.
struct StripCtl {
  uint64_t key;     // local maximum as (score, -row, -column)
  int32_t flags;    // 1 invalid residue, 2 a wait ran out
  int32_t done;     // strips finished
  int32_t last_h;   // H(m, n)
  int32_t pad[3];
};
static_assert(sizeof(StripCtl) == 32, "record size");

// A warp task: up to 32/G pairs of one lane width G, processed by one warp
// (x = first index into the task list, y = (G << 16) | number of pairs).
// The planner orders warp tasks longest first; warps of one persistent
// launch pull them from a single counter.
struct FillArgs {
  const uint8_t *codes;
  const PairDev *pairs;
  const int32_t *tasks;  // pair ids, grouped by warp task
  const int2 *wtasks;
  int32_t n_wtasks;
  const int32_t *n_wtasks_dev;  // when set, the warp-task count is read here (int32 re-run)
  int32_t *counter;      // work-queue head, zero before the launch
  const int8_t *matrix;  // 26*26 device copy of the scheme
  int32_t gap_open, gap_extend;
  ResultDev *res;
  int32_t *bnd;          // boundary scratch: per warp, 8 group rows
  int32_t bnd_cols;      // entries per group row (max n over the launch, even)
  uint8_t *planes;       // TB planes (kOutTrace)
  const int64_t *plane_off;  // byte offset of each pair's planes
  int32_t *overflow;     // int16 CHECK: per pair, 1 when a lane came near 32767
  int32_t max_score;     // largest substitution score of the scheme
  int32_t min_score;     // smallest
  uint32_t one;          // int16x2 fill: 1, an opaque multiplier for packed subtractions on the IMAD pipe
  const uint8_t *ccodes;  // int16x2 fill: class code per residue (0 for invalid ones), same offsets as codes
  const int8_t *cmatrix;  // int16x2 fill: nclasses x nclasses class scores
  int32_t nclasses;
  int32_t spin_limit;     // CTA and strip fills: polls per bounded wait (0 = the compiled default)
  // Strip fills (wtasks lists (position in tasks, strip); null: one pair's
  // strips in order): per pair of the launch, a record and its hand-over row
  // (both zero before the launch).
  StripCtl *strip_ctl;
  uint64_t *strip_rows;
  const int64_t *strip_row_off;  // entries
};

// Compacts the pairs an int16 CHECK launch flagged into a warp-task list
// for the int32 re-run (one pair per warp task, same lane width).
cudaError_t launch_collect_overflow(const int32_t *checked, int32_t n_checked, const int32_t *overflow,
                                    const int32_t *pair_g, int32_t *rerun_tasks, int2 *rerun_wtasks,
                                    int32_t *rerun_count, cudaStream_t st);

struct WalkArgs {
  const uint8_t *seqs;  // ASCII residues (for the emitted strings)
  const uint8_t *codes;
  const PairDev *pairs;
  const int32_t *tasks;
  int32_t n_tasks;
  const uint8_t *planes;
  const int64_t *plane_off;
  const int32_t *shape_G;  // per pair: the G and R its planes were written with
  const int32_t *shape_R;
  int32_t local;
  int32_t emit;  // 0: counts only (no rows, no local begin coordinates)
  ResultDev *res;
  char *aln;                 // per pair: 2 * cap bytes (a row then b row)
  const int64_t *aln_off;
  int32_t skip_begin, skip_end;  // launch_walk: tasks that another launch walks
  // launch_walk_block: per task, the pair's row (strip_row_entries), for the
  // path's records of pairs whose records do not fit shared memory.
  uint64_t *rec_rows;
  const int64_t *rec_off;
  int32_t rec_words;
};

// Host-side helpers (scheme.cpp).
int build_scheme(const tsq_params *p, Scheme *out);
// BLOSUM62 entry by row index in the order ARNDCQEGHILKMFPSTWYVBZX.
int8_t blosum62_by_row(int x, int y);
void build_lut(const Scheme &s, uint8_t lut[256]);
// Byte -> score class (0 for bytes the scheme rejects, which their letter
// code marks invalid).
void build_class_lut(const Scheme &s, uint8_t lut[256]);

// A launch that may (early) start before the one ahead of it in the stream ends.
template <class Args>
cudaError_t launch_maybe_early(void (*kernel)(const Args), dim3 grid, int threads, size_t smem, cudaStream_t st,
                               bool early, const Args &args) {
  cudaLaunchAttribute attr[1] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

// Kernel launchers (fill_dispatch.cu, fill_i16.cu, fill_cta.cu, walk_kernel.cu).
// Returns the number of thread blocks a persistent launch of this shape uses.
// A launch covers every lane width G of one row height R and lane type
// (i16: 0 int32, 1 int16x2, 2 int16x2 with overflow check).
// Blocks of a fill launch resident on the device; nclasses sizes the int16x2
// fill's profile (ignored by the int32 fills).
int fill_blocks(int R, int i16, int out_mode, bool local, int nclasses = kLetters);
size_t fill_smem_bytes(int R, int i16, int out_mode, int nclasses = kLetters);
int fill_threads();
int fill_threads_for(int i16);
size_t fill_bnd_entry_bytes(int i16, int out_mode);
cudaError_t launch_fill(int R, int i16, int out_mode, bool local, const FillArgs &a, int blocks,
                        cudaStream_t st);
bool shape_supported(const Shape &sh, int out_mode, bool local);
// One long pair per CTA (fill_cta.cu): identity output.  FillArgs.tasks /
// n_wtasks hold the pair list, bnd one wrap-around row of bnd_cols entries
// per block.
int cta_blocks(bool local);
size_t cta_bnd_entry_bytes();
cudaError_t launch_cta(bool local, const FillArgs &a, int blocks, cudaStream_t st);
// One pair spread over the GPU's warps in strips of rows (fill_strip.cu):
// score and traceback output, in int32 lanes (strips of 128 rows) or int16x2
// lanes with rebased values (512 rows; open + ext + max_score <= 40).
// FillArgs carries the class codes, class matrix and class count, the unit
// list and the strip workspace.
enum StripKind : int { kStrip32 = 0, kStrip16 = 1 };
bool strip16_supported(const Scheme &sc, int32_t gap_open, int32_t gap_extend);
int strip_rows(StripKind kind);
Shape strip_shape(StripKind kind);  // of the traceback planes
int strip_blocks(StripKind kind, int out_mode, bool local, int nclasses);
// early: may start before the launch ahead of it in the stream ends (which must
// be one that lets it: launch_encode, launch_strip); the kernel waits for it.
cudaError_t launch_strip(StripKind kind, int out_mode, bool local, const FillArgs &a, int blocks, cudaStream_t st,
                         bool early = false);
// The work of a set of pairs in each kind of strips, and the kind that is
// estimated to finish first: the longer of its longest pair's chain of steps
// and its total steps over all schedulers.
struct StripLoad {
  double steps[2] = {0.0, 0.0}, chain[2] = {0.0, 0.0};
  void add(int m, int n);
  void merge(const StripLoad &o);
  StripKind pick(int out_mode, int sms, bool allow16) const;
};
cudaError_t launch_walk(const WalkArgs &a, cudaStream_t st);
// The pairs of a strip launch, one block each; max_rows: their longest a.
// Pairs of at least kWalkRecRows rows need room for their records.
constexpr int32_t kWalkRecRows = 32768;
// 64-bit entries of a pair's row in global memory in strips of `rows` rows: its
// n hand-over entries where there is more than one strip; walked pairs of
// kWalkRecRows rows and more keep the walk's 32-bit records of rows 0 to m there
// afterwards.  In whole 128 bytes.
inline int64_t strip_row_entries(int32_t m, int32_t n, int rows, bool walk) {
  int64_t entries = m > rows ? n : 0;
  if (walk && m >= kWalkRecRows) entries = std::max<int64_t>(entries, (int64_t(m) + 2) / 2);
  return (entries + 15) & ~int64_t(15);
}
cudaError_t launch_walk_block(const WalkArgs &a, int R, int32_t max_rows, cudaStream_t st, bool early = false);
// Residues -> letter codes and, when clut_dev / ccodes are set, score
// classes.
// zero: zero_bytes (a multiple of 16, 16-byte aligned) that the launch also clears.
cudaError_t launch_encode(const uint8_t *seqs, int64_t len, const uint8_t *lut_dev, uint8_t *codes,
                          const uint8_t *clut_dev, uint8_t *ccodes, cudaStream_t st,
                          void *zero = nullptr, int64_t zero_bytes = 0);

// Bytes of traceback planes a pair needs under a shape: words of eight cells
// per lane, R rows (8, or 4 in int32 strips) of 8 / R steps (step = column +
// lane).
inline int64_t plane_bytes(int m, int n, const Shape &sh) {
  if (m <= 0 || n <= 0) return 0;
  const int64_t P = (int64_t)sh.G * sh.R, U = 8 / sh.R;
  const int64_t bands = (m + P - 1) / P;
  return (bands * ((n + sh.G - 1 + U - 1) / U) * sh.G * 4 + 15) & ~int64_t(15);
}

}  // namespace tsq
