// fill_strip.cu -- instantiations, launcher and choice of the strip fills.
#include <map>
#include <mutex>
#include <tuple>

#include "fill_strip16.cuh"
#include "fill_strip32.cuh"

namespace tsq {
namespace fill {
namespace {

using Kernel = void (*)(const FillArgs);

template <int OUT, bool LOCAL>
Kernel kernel_of(StripKind kind) {
  return kind == kStrip16 ? fill_strip16_kernel<OUT, LOCAL> : fill_strip32_kernel<OUT, LOCAL>;
}

Kernel strip_kernel(StripKind kind, int out_mode, bool local) {
  if (out_mode == kOutTrace) return local ? kernel_of<kOutTrace, true>(kind) : kernel_of<kOutTrace, false>(kind);
  if (out_mode == kOutScore) return local ? kernel_of<kOutScore, true>(kind) : kernel_of<kOutScore, false>(kind);
  return nullptr;
}

size_t strip_smem(StripKind kind, int nclasses) {
  return kind == kStrip16 ? strip16_smem_bytes(nclasses) : strip32_smem_bytes(nclasses);
}

// What a kind's steps cost, in cycles [score, traceback]: on a scheduler with
// no other warp (a lone pair's chain of steps; measured on 1 x 20,000) and on
// a full one (per warp step; 64 x 30,000); and the steps between the starts
// of two consecutive strips.
struct Cost {
  int rows, ramp;
  double lag, alone[2], full[2];
};
const Cost &cost_of(StripKind kind) {
  static const Cost costs[2] = {
      {kStripRows32, 31, 70.0, {118.0, 175.0}, {89.0, 159.0}},
      {kStripRows16, 63, 100.0, {175.0, 365.0}, {150.0, 300.0}},
  };
  return costs[kind];
}

}  // namespace
}  // namespace fill

bool strip16_supported(const Scheme &sc, int32_t gap_open, int32_t gap_extend) {
  const int64_t step = int64_t(gap_open) + gap_extend + std::max(sc.max_score, 0);
  return step <= fill::kMaxStep16 && sc.min_score >= -128 && sc.nclasses >= 1 && sc.nclasses <= kLetters;
}

int strip_rows(StripKind kind) { return fill::cost_of(kind).rows; }
Shape strip_shape(StripKind kind) { return Shape{32, kind == kStrip16 ? 8 : strip_rows(kind) / 32, 0}; }

void StripLoad::add(int m, int n) {
  if (m <= 0 || n <= 0) return;
  for (int k = 0; k < 2; ++k) {
    const fill::Cost &c = fill::cost_of(StripKind(k));
    const double strips = double((m + c.rows - 1) / c.rows), sweep = double(n) + c.ramp;
    steps[k] += strips * sweep;
    chain[k] = std::max(chain[k], sweep + (strips - 1.0) * c.lag);
  }
}

void StripLoad::merge(const StripLoad &o) {
  for (int k = 0; k < 2; ++k) {
    steps[k] += o.steps[k];
    chain[k] = std::max(chain[k], o.chain[k]);
  }
}

StripKind StripLoad::pick(int out_mode, int sms, bool allow16) const {
  const int tr = out_mode == kOutTrace ? 1 : 0;
  StripKind best = kStrip32;
  double best_t = 0.0;
  for (int k = 0; k < (allow16 ? 2 : 1); ++k) {
    const fill::Cost &c = fill::cost_of(StripKind(k));
    const double t = std::max(chain[k] * c.alone[tr], steps[k] * c.full[tr] / (4.0 * sms));
    if (k == 0 || t < best_t) {
      best = StripKind(k);
      best_t = t;
    }
  }
  return best;
}

// Blocks (warps) of a strip launch: two on each scheduler, one beside other fills.
// Device time of the fills, ms, with as many as fit (2.5 a scheduler and more,
// unevenly spread) / two / one: 23 DNA pairs of 10 to 50 kb with traceback 25.0 /
// 22.8 / 24.2, score 11.3 / 10.8 / 12.3, 200 of 3 to 9 kb 5.6 / 5.1 / 5.8; strips
// beside short pairs, 1,000 proteins of median 800 1.48 / 1.48 / 1.05, 60 of median
// 4,000 5.1 / 3.7 / 3.4.  Two warps fill a scheduler; a third only lengthens the
// steps of the longest pair's chain, and an uneven spread lengthens some.
int strip_blocks(StripKind kind, int out_mode, bool local, int nclasses) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, bool, int>, int> known;
  const auto key = std::make_tuple(dev, int(kind), out_mode, local, nclasses);
  {
    std::lock_guard<std::mutex> g(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const fill::Kernel k = fill::strip_kernel(kind, out_mode, local);
  int nb = 0;
  constexpr int kSchedulers = 4;
  if (!k || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, 32, fill::strip_smem(kind, nclasses)) != cudaSuccess)
    return 0;
  nb = std::min(nb, 2 * kSchedulers);
  if (nb * sms > 0) {
    std::lock_guard<std::mutex> g(mu);
    known[key] = nb * sms;
  }
  return nb * sms;
}

cudaError_t launch_strip(StripKind kind, int out_mode, bool local, const FillArgs &args, int blocks, cudaStream_t st,
                         bool early) {
  const fill::Kernel k = fill::strip_kernel(kind, out_mode, local);
  if (!k) return cudaErrorInvalidValue;
  FillArgs a = args;
  a.one = 1u;
  return launch_maybe_early(k, dim3(blocks), 32, fill::strip_smem(kind, a.nclasses), st, early, a);
}

}  // namespace tsq
