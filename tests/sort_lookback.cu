// The sort's look-back (voxel_b200/csrc/sort_lookback.cuh) of one tile, by one
// block, over words that the test writes.
#include "../voxel_b200/csrc/sort_lookback.cuh"

namespace {
__global__ void lookback_kernel(vx::sort::Records r, uint32_t tile, uint32_t count,
                                uint32_t *exclusive, uint32_t *status) {
  exclusive[threadIdx.x] = vx::sort::digit_lookback(r, tile, threadIdx.x, count, status);
}
} // namespace

extern "C" uint32_t lookback_rows(uint32_t tiles) { return vx::sort::record_rows(tiles); }

extern "C" int lookback(uint32_t *words, uint32_t tiles, uint32_t tile, uint32_t count,
                        uint32_t *exclusive, uint32_t *status) {
  lookback_kernel<<<1, vx::sort::kBins>>>(vx::sort::records_of(words, tiles), tile, count,
                                          exclusive, status);
  return static_cast<int>(cudaDeviceSynchronize());
}
