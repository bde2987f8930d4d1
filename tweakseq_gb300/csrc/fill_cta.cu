// fill_cta.cu -- instantiations of the CTA-per-pair int32 identity fill.
#include <map>
#include <mutex>
#include <tuple>

#include "fill_cta.cuh"

namespace tsq {
namespace fill {
namespace {

constexpr int kW = 8;  // warps per CTA: the path counts' registers do not fit 16

int occ(bool local) {
  const size_t smem = cta_smem_bytes(kW);
  auto k = local ? fill_cta_kernel<true, kW> : fill_cta_kernel<false, kW>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kW * 32, smem) != cudaSuccess) return 0;
  return nb;
}

}  // namespace
}  // namespace fill

// Resident CTAs of the long-pair fill on the current device (occupancy
// queries cached per device and kernel, as for the warp fills).
int cta_blocks(bool local) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  static std::mutex mu;
  static std::map<std::tuple<int, int>, int> known;
  const auto key = std::make_tuple(dev, int(local));
  {
    std::lock_guard<std::mutex> g(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = fill::occ(local) * sms;
  if (blocks > 0) {
    std::lock_guard<std::mutex> g(mu);
    known[key] = blocks;
  }
  return blocks;
}

size_t cta_bnd_entry_bytes() { return 16; }

cudaError_t launch_cta(bool local, const FillArgs &a, int blocks, cudaStream_t st) {
  const size_t smem = fill::cta_smem_bytes(fill::kW);
  if (local)
    fill::fill_cta_kernel<true, fill::kW><<<blocks, fill::kW * 32, smem, st>>>(a);
  else
    fill::fill_cta_kernel<false, fill::kW><<<blocks, fill::kW * 32, smem, st>>>(a);
  return cudaGetLastError();
}

}  // namespace tsq
