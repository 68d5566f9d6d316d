// Look-back of the radix sort's partition passes over the digit counts of
// earlier tiles (sort.cu).
#pragma once

#include "common.cuh"

namespace vx::sort {

constexpr uint32_t kRadixBits = 8; // the widest digit (256 counters per table)
constexpr uint32_t kBins = 1u << kRadixBits;

// Look-back words, one per digit each (the block's threads are the digits):
//   per tile: its count under a ready bit;
//   per group of 8 tiles and per super-group of 64: the sum of the counts
//     plus the number of tiles << 24 (64 tiles of 4,096 keys sum below 2^24);
//   per super-group: the inclusive count over all tiles up to its last one,
//     under a ready bit.
constexpr uint32_t kReady = 1u << 31;
constexpr uint32_t kGroup = 8, kSuper = 64, kTiles = 24;
constexpr uint32_t kSumMask = (1u << kTiles) - 1u;
struct Records {
  uint32_t *tile, *group, *super, *inclusive; // [...][256]
};
inline uint32_t record_rows(uint32_t tiles) {
  return tiles + ceil_div(tiles, kGroup) + 2u * ceil_div(tiles, kSuper);
}
inline Records records_of(uint32_t *words, uint32_t tiles) {
  Records r;
  r.tile = words;
  r.group = r.tile + static_cast<size_t>(tiles) * 256u;
  r.super = r.group + static_cast<size_t>(ceil_div(tiles, kGroup)) * 256u;
  r.inclusive = r.super + static_cast<size_t>(ceil_div(tiles, kSuper)) * 256u;
  return r;
}

// Thread t publishes the tile's count of digit t.
__device__ __forceinline__ void publish_count(const Records &r, uint32_t tile, uint32_t t,
                                              uint32_t count) {
  st_relaxed_u32(r.tile + static_cast<size_t>(tile) * kBins + t, kReady | count);
  atomicAdd(r.group + static_cast<size_t>(tile / kGroup) * kBins + t, (1u << kTiles) | count);
  atomicAdd(r.super + static_cast<size_t>(tile / kSuper) * kBins + t, (1u << kTiles) | count);
}

// The GPU timer in units of 65.5 us, for a look-back's limit: a 32-bit word
// that is read once costs the passes nothing, a 64-bit one that the first wait
// sets 1-2 % at 1 M keys.
constexpr uint32_t kTickShift = 16;
__device__ __forceinline__ uint32_t timer_ticks() {
  return static_cast<uint32_t>(global_ns() >> kTickShift);
}

// Reads *p until ready(value); `v` is the value read already.  All waits of a
// look-back that began at `began` share one limit: once it has run out, a word
// that is not there on the next read counts as 0.
template <class Ready>
__device__ __forceinline__ uint32_t wait_word(const uint32_t *p, uint32_t v, Ready ready,
                                              uint32_t began, uint32_t *status) {
  if (ready(v)) return v;
  for (;;) {
    __nanosleep(20);
    v = ld_relaxed_u32(p);
    if (ready(v)) return v;
    if (timer_ticks() - began > static_cast<uint32_t>(kWaitLimitNs >> kTickShift)) {
      set_status(status, kDevTimeout);
      return 0;
    }
  }
}

// Per-digit look-back, once every tile publishes with publish_count: the sum
// of the tiles before this one in its group, of the groups before it in its
// super-group, and of the super-groups back to the nearest inclusive count
// (the last tile of a super-group publishes that one, so the smallest
// unfinished tile always finds its predecessor's).  The words of the first
// round are read together; afterwards only a word that is not there yet is
// read again.  Reading eight tiles a round trip back to an inclusive one took
// a dozen rounds with ~600 tiles in flight, ~100 of a pass's 169 instructions
// per u64 key.  Returns the digit's count over all earlier tiles; after a
// timeout (*status is set) what was there of it, which is never more.
__device__ __forceinline__ uint32_t digit_lookback(const Records &r, uint32_t tile, uint32_t t,
                                                   uint32_t tile_count, uint32_t *status) {
  constexpr uint32_t kFirst = 4; // super-groups read in the first round
  const uint32_t in = tile % kGroup, group = tile / kGroup, gin = group % (kSuper / kGroup);
  const uint32_t super = tile / kSuper;
  const uint32_t *tiles = r.tile + static_cast<size_t>(tile - in) * kBins + t;
  const uint32_t *groups = r.group + static_cast<size_t>(group - gin) * kBins + t;
  auto row = [&](const uint32_t *words, uint32_t i) {
    return words + static_cast<size_t>(i) * kBins + t;
  };
  uint32_t own[kGroup - 1], grp[kSuper / kGroup - 1], sum[kFirst], inc[kFirst];
#pragma unroll
  for (uint32_t j = 0; j < kGroup - 1; ++j)
    own[j] = j < in ? ld_relaxed_u32(tiles + j * kBins) : 0u;
#pragma unroll
  for (uint32_t j = 0; j < kSuper / kGroup - 1; ++j)
    grp[j] = j < gin ? ld_relaxed_u32(groups + j * kBins) : 0u;
#pragma unroll
  for (uint32_t j = 0; j < kFirst; ++j) {
    inc[j] = super > j ? ld_relaxed_u32(row(r.inclusive, super - 1 - j)) : 0u;
    sum[j] = super > j ? ld_relaxed_u32(row(r.super, super - 1 - j)) : 0u;
  }
  auto tile_ready = [](uint32_t v) { return (v & kReady) != 0; };
  auto group_ready = [](uint32_t v) { return (v >> kTiles) == kGroup; };
  auto super_ready = [](uint32_t v) { return (v >> kTiles) == kSuper; };
  const uint32_t began = timer_ticks();
  auto wait = [&](const uint32_t *p, uint32_t v, auto ready) {
    return wait_word(p, v, ready, began, status);
  };
  uint32_t exclusive = 0;
  bool found = super == 0;
#pragma unroll
  for (uint32_t j = 0; j < kFirst; ++j) {
    if (found || super <= j) continue;
    if (inc[j] & kReady) {
      exclusive += inc[j] & ~kReady;
      found = true;
    } else {
      exclusive += wait(row(r.super, super - 1 - j), sum[j], super_ready) & kSumMask;
      found = super == j + 1; // the first super-group: nothing before it
    }
  }
  for (uint32_t k = super - 1 - kFirst; !found; --k) { // (super > kFirst here)
    const uint32_t v = ld_relaxed_u32(row(r.inclusive, k));
    const uint32_t w = ld_relaxed_u32(row(r.super, k));
    if (v & kReady) {
      exclusive += v & ~kReady;
      found = true;
    } else {
      exclusive += wait(row(r.super, k), w, super_ready) & kSumMask;
      found = k == 0;
    }
  }
#pragma unroll
  for (uint32_t j = 0; j < kSuper / kGroup - 1; ++j)
    if (j < gin) exclusive += wait(groups + j * kBins, grp[j], group_ready) & kSumMask;
#pragma unroll
  for (uint32_t j = 0; j < kGroup - 1; ++j)
    if (j < in) exclusive += wait(tiles + j * kBins, own[j], tile_ready) & ~kReady;
  if (tile % kSuper == kSuper - 1)
    st_relaxed_u32(r.inclusive + static_cast<size_t>(super) * kBins + t,
                   kReady | (exclusive + tile_count));
  return exclusive;
}

} // namespace vx::sort
