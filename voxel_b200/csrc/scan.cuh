// Single-pass prefix sum with decoupled look-back (Merrill & Garland 2016,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back"), written for
// sm_100a: each tile arrives in shared memory by one bulk copy (TMA), a
// dynamic tile id makes a tile only ever wait on tiles that are already
// resident, a tile's 32-bit sum also goes into the sum of its group of 32
// tiles, so that one round trip of three loads per lane reads 1,024
// predecessors, and a globaltimer bound limits every wait.
//
// Replaces the reference's BlockBased<DecoupledLookback<WarpShuffleBlock<512,4>>>
// (cuda/scan/block_based/decoupled_lookback.cuh:116-221), whose look-back is a
// single thread with an unbounded spin (:99-102), and its fused variant
// (cuda/scan/fused.cuh:102-159), which assumes in-order block scheduling.
#pragma once

#include "common.cuh"

namespace vx::scan {

// Look-back record states.
constexpr uint32_t kNotReady = 0, kAggregate = 1, kInclusive = 2;

// u32 sums: a tile's record is its sum under a ready bit, one relaxed 64-bit
// store.  The tile also adds its sum and 1 << kGroupCount to the word of its
// group (32 tiles: the sums stay below the count), so a word whose count is 32
// holds the whole group's sum; the group's last tile writes the group's
// inclusive prefix, again under a ready bit.
struct GroupRecords32 {
  uint64_t *tile;
  uint64_t *group_sum;
  uint64_t *group_inc;
};
constexpr uint32_t kGroup = 32, kGroupCount = 40;
constexpr uint64_t kReady = 1ull << 63;

__device__ __forceinline__ void publish_group(const GroupRecords32 &r, uint32_t tile,
                                              uint32_t aggregate) {
  atomicAdd(reinterpret_cast<unsigned long long *>(r.group_sum + tile / kGroup),
            (1ull << kGroupCount) + aggregate);
  st_relaxed_u64(r.tile + tile, kReady | aggregate);
}

// Look-back for u32 sums, called by one full warp after lane 0 published the
// tile (publish_group): lane l reads the record of its group's tile l and the
// words of the l-th group back, until the tiles before it in its group and the
// groups back to the nearest inclusive prefix are all there; a lane reads
// again only what it has not got.  The smallest unfinished tile always finds
// the inclusive prefix of the group before its own, so every tile ends.
// Returns the sum of all earlier tiles (in every lane); on timeout sets
// *status and returns a partial sum.
__device__ __forceinline__ uint32_t group_lookback(const GroupRecords32 &r, uint32_t tile,
                                                   uint32_t aggregate, uint32_t *status) {
  const uint32_t lane = lane_id();
  const uint32_t group = tile / kGroup, in = tile % kGroup;
  const int64_t g = static_cast<int64_t>(group) - 1 - lane;
  uint64_t own = lane < in ? 0ull : kReady;
  uint64_t sum = 0, inc = g < 0 ? kReady : 0ull; // nothing before the first group
  uint32_t exclusive = 0;
  uint64_t t0 = 0;
  for (;;) {
    if (!(own & kReady)) own = ld_relaxed_u64(r.tile + group * kGroup + lane);
    if (!(inc & kReady)) {
      inc = ld_relaxed_u64(r.group_inc + g);
      if ((sum >> kGroupCount) != kGroup) sum = ld_relaxed_u64(r.group_sum + g);
    }
    const bool own_all = __all_sync(kFullMask, (own & kReady) != 0);
    const uint32_t found = __ballot_sync(kFullMask, (inc & kReady) != 0);
    const uint32_t whole = __ballot_sync(kFullMask, (sum >> kGroupCount) == kGroup);
    const uint32_t nearest = found ? __ffs(found) - 1u : 0u;
    const uint32_t between = (1u << nearest) - 1u;
    const bool there = own_all && found && (whole & between) == between;
    if (there || (t0 != 0 && global_ns() - t0 > kWaitLimitNs)) {
      if (!there && lane == 0) set_status(status, kDevTimeout);
      uint32_t v = lane < in ? static_cast<uint32_t>(own) : 0u;
      if (lane < nearest) v += static_cast<uint32_t>(sum);
      else if (lane == nearest) v += static_cast<uint32_t>(inc);
      exclusive = __reduce_add_sync(kFullMask, v);
      break;
    }
    if (t0 == 0) t0 = global_ns();
  }
  if (in == kGroup - 1u && lane == 0)
    st_relaxed_u64(r.group_inc + group, kReady | (exclusive + aggregate));
  return exclusive;
}

// u64 sums keep the value beside a state word: value first, then a release
// store of the state; readers acquire the state before reading the value.
struct SplitRecords64 {
  uint64_t *agg;
  uint64_t *inc;
  uint32_t *state;
  __device__ void publish(uint32_t tile, uint32_t s, uint64_t value) const {
    st_relaxed_u64((s == kInclusive ? inc : agg) + tile, value);
    st_release_u32(state + tile, s);
  }
  __device__ void read(int64_t tile, uint32_t &s, uint64_t &value) const {
    if (tile < 0) {
      s = kInclusive;
      value = 0;
      return;
    }
    s = ld_acquire_u32(state + tile);
    value = s == kInclusive ? ld_relaxed_u64(inc + tile)
                            : (s == kAggregate ? ld_relaxed_u64(agg + tile) : 0);
  }
};

template <class T> struct RecordsFor;
template <> struct RecordsFor<uint32_t> { using type = GroupRecords32; };
template <> struct RecordsFor<uint64_t> { using type = SplitRecords64; };

// Warp-parallel look-back for u64 sums, called by one full warp after lane 0
// published the tile's aggregate (SplitRecords64::publish).  Reads the records
// of the previous 32 * R tiles at once (lane l, row j reads distance l + 32 j:
// R coalesced loads in flight per lane), accumulates back to the nearest
// inclusive record, publishes the inclusive prefix and returns the exclusive
// prefix (valid in every lane).
// A window wider than one warp matters because with hundreds of tiles
// resident the nearest inclusive record can be far back, and each window
// costs one round trip to L2.  On timeout sets *status and returns a partial
// sum.
template <class T, uint32_t R = 2, class Records>
__device__ T warp_lookback(const Records &records, uint32_t tile, T aggregate,
                           uint32_t *status) {
  const uint32_t lane = lane_id();
  if (tile == 0) return T(0);
  T exclusive = 0;
  int64_t pos = static_cast<int64_t>(tile) - 1;
  const uint64_t t0 = global_ns();
  for (;;) {
    uint32_t st[R];
    T v[R];
#pragma unroll
    for (uint32_t j = 0; j < R; ++j)
      records.read(pos - static_cast<int64_t>(lane + kWarp * j), st[j], v[j]);
    // Nearest inclusive record: first row with one, first lane in it.
    int32_t first_row = -1;
    uint32_t limit = 31;
    bool wait = false;
#pragma unroll
    for (uint32_t j = 0; j < R; ++j) {
      const uint32_t inc = __ballot_sync(kFullMask, st[j] == kInclusive);
      const uint32_t nr = __ballot_sync(kFullMask, st[j] == kNotReady);
      if (first_row < 0) {
        const uint32_t lim = inc ? (__ffs(inc) - 1u) : 31u;
        const uint32_t range = lim == 31u ? kFullMask : ((1u << (lim + 1u)) - 1u);
        wait = wait || (nr & range) != 0;
        if (inc) {
          first_row = static_cast<int32_t>(j);
          limit = lim;
        }
      }
    }
    if (wait) {
      if (global_ns() - t0 > kWaitLimitNs) {
        if (lane == 0) set_status(status, kDevTimeout);
        break;
      }
      __nanosleep(32);
      continue;
    }
    T part = 0;
#pragma unroll
    for (uint32_t j = 0; j < R; ++j) {
      const bool in = first_row < 0 || static_cast<int32_t>(j) < first_row ||
                      (static_cast<int32_t>(j) == first_row && lane <= limit);
      part += in ? v[j] : T(0);
    }
    exclusive += warp_sum<T>(part);
    if (first_row >= 0) break;
    pos -= static_cast<int64_t>(kWarp * R);
  }
  if (lane == 0) records.publish(tile, kInclusive, exclusive + aggregate);
  return exclusive;
}

// Tile geometry: Block threads x Rows rows of 16-byte vectors, each warp a
// contiguous part of the tile.  The tile is staged in shared memory by one
// bulk copy and read from there twice (sums, then prefix sums), so a thread
// keeps one value per row.  What bounds the bandwidth is the bytes in flight
// per SM while tiles wait for their loads and for the tiles before them:
// shared memory holds six 32 KB tiles.  On B200, 2^27 u32 (1.07 GB), 164 us at
// the measured copy bandwidth:
//   look-back over 64 tile records per round trip, rows scanned before the
//     tile's sum is published (256 threads)                          301 us
//   sum published first, rows scanned while the records are on the way 279 us
//   group sums as above, 256 threads x 8 rows, 6 per SM              225 us
//   the same, 128 threads x 16 rows, 6 per SM (this shape)       217-225 us
//   48 KB tiles, 4 per SM 214 us; 64 KB, 3 per SM 223 us; 16 KB, 12 per SM
//   250 us (more tiles: more round trips).
// The "scan.tile_kb" knob offers 16 and 8 KB tiles.
template <class T, uint32_t Block = 128, uint32_t Rows = 16, uint32_t MinBlocks = 6>
struct TileShape {
  static constexpr uint32_t kBlock = Block;
  static constexpr uint32_t kRows = Rows;
  static constexpr uint32_t kMinBlocks = MinBlocks;
  static constexpr uint32_t kPerVec = 16 / sizeof(T);
  static constexpr uint32_t kTile = kBlock * kRows * kPerVec;
  static constexpr uint32_t kWarps = kBlock / kWarp;
};
template <class T> using Tile32 = TileShape<T>;
template <class T> using Tile16 = TileShape<T, 128, 8, 12>;
template <class T> using Tile8 = TileShape<T, 64, 8, 24>;

struct ScanLayout {
  uint32_t *tile_counter;
  uint32_t *status;
  uint64_t *rec_a;
  uint64_t *rec_b;
  uint32_t *rec_state;
};

size_t workspace_size(uint32_t count);
ScanLayout carve(void *workspace, uint32_t count);

template <class T>
vx_status scan_launch(T *data, uint32_t count, bool inclusive, void *workspace,
                      size_t workspace_bytes, cudaStream_t stream);

} // namespace vx::scan
