// In-place prefix sums (uint32 / uint64, wrapping), one kernel launch after a
// small memset of the look-back records.  See scan.cuh for the design.
#include "profile.cuh"
#include "scan.cuh"
#include "tuning.cuh"

#include <cuda.h>

#include <mutex>

namespace vx {

int sm_count() {
  static int cached = 0;
  if (cached == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev);
    if (cached <= 0) cached = 148;
  }
  return cached;
}

namespace scan {

namespace {

inline uint32_t groups_of(uint32_t tiles) { return ceil_div(tiles, kGroup); }

// The records of `tiles` tiles: u32 sums keep a word per tile and two per
// group in a row, u64 sums three arrays.  *end: the first byte after what a
// call has to clear.
template <class T>
typename RecordsFor<T>::type make_records(const ScanLayout &ws, uint32_t tiles, char **end) {
  typename RecordsFor<T>::type r;
  if constexpr (sizeof(T) == 4) {
    r.tile = ws.rec_a;
    r.group_sum = r.tile + tiles;
    r.group_inc = r.group_sum + groups_of(tiles);
    *end = reinterpret_cast<char *>(r.group_inc + groups_of(tiles));
  } else {
    r.agg = ws.rec_a;
    r.inc = ws.rec_b;
    r.state = ws.rec_state;
    *end = reinterpret_cast<char *>(ws.rec_state + tiles);
  }
  return r;
}

// One tile per block, tiles taken in the order of a global counter (a tile
// only waits on tiles already taken by running blocks).  A full, aligned tile
// arrives by one bulk copy; the last, partial tile and unaligned data use
// guarded loads.  Each warp owns a contiguous part of the tile: it sums its
// rows, the tile's sum is published at once, and while warp 0 looks back the
// rows are scanned (32 lanes' vectors a row); then the rows are read from
// shared memory again and the prefix sums written straight to global memory.
template <class T, bool Inclusive, bool Vectorised, class S = Tile32<T>>
__global__ void __launch_bounds__(S::kBlock, S::kMinBlocks)
    scan_kernel(T *__restrict__ data, uint32_t count, ScanLayout ws,
                typename RecordsFor<T>::type records) {
  constexpr uint32_t kTileBytes = S::kTile * sizeof(T);
  __shared__ __align__(128) T s_data[S::kTile];
  __shared__ uint64_t s_bar;
  __shared__ uint32_t s_tile;
  __shared__ T s_warp[S::kWarps];
  __shared__ T s_prefix;

  const uint32_t t = threadIdx.x;
  const uint32_t lane = lane_id();
  const uint32_t warp = t / kWarp;
  if (t == 0) {
    const uint32_t tile = atomicAdd(ws.tile_counter, 1u);
    s_tile = tile;
    if (Vectorised && static_cast<uint64_t>(tile + 1) * S::kTile <= count) {
      mbar_init(&s_bar, 1);
      mbar_arrive_expect_tx(&s_bar, kTileBytes);
      bulk_load(s_data, data + static_cast<uint64_t>(tile) * S::kTile, kTileBytes, &s_bar);
    }
  }
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = static_cast<uint64_t>(tile) * S::kTile;
  const bool bulk = Vectorised && base + S::kTile <= count;
  if (bulk) {
    if (!mbar_wait(&s_bar, 0)) {
      // Never expected: report, let the copy land, give up on this tile.
      if (t == 0) set_status(ws.status, kDevTimeout);
      mbar_wait(&s_bar, 0);
      return;
    }
  } else {
    for (uint32_t i = t; i < S::kTile; i += S::kBlock)
      s_data[i] = base + i < count ? data[base + i] : T(0);
    __syncthreads();
  }
  const uint32_t first_vec = warp * S::kRows * kWarp + lane; // row r: first_vec + 32 r
  const uint4 *vecs = reinterpret_cast<const uint4 *>(s_data);

  // The lane's sum in each row, and the tile's sum.
  T at[S::kRows];
  T total = 0;
#pragma unroll
  for (uint32_t r = 0; r < S::kRows; ++r) {
    const uint4 q = vecs[first_vec + r * kWarp];
    const T *qt = reinterpret_cast<const T *>(&q);
    T sum = 0;
#pragma unroll
    for (uint32_t e = 0; e < S::kPerVec; ++e) sum += qt[e];
    at[r] = sum;
    total += sum;
  }
  total = warp_sum<T>(total);
  if (lane == 0) s_warp[warp] = total;
  __syncthreads();
  T aggregate = 0, run = 0; // of the tile, of the warps before this one
#pragma unroll
  for (uint32_t w = 0; w < S::kWarps; ++w) {
    const T v = s_warp[w];
    if (w < warp) run += v;
    aggregate += v;
  }
  if (t == 0) {
    if constexpr (sizeof(T) == 4) publish_group(records, tile, aggregate);
    else records.publish(tile, tile == 0 ? kInclusive : kAggregate, aggregate);
  }
  if (warp == 0) {
    T prefix;
    if constexpr (sizeof(T) == 4) prefix = group_lookback(records, tile, aggregate, ws.status);
    else prefix = warp_lookback<T>(records, tile, aggregate, ws.status);
    if (lane == 0) s_prefix = prefix;
  }
  // Each lane's offset in the tile, row by row.
#pragma unroll
  for (uint32_t r = 0; r < S::kRows; ++r) {
    const T inc = warp_inclusive_sum<T>(at[r]);
    const T row = __shfl_sync(kFullMask, inc, kWarp - 1);
    at[r] = run + inc - at[r];
    run += row;
  }
  __syncthreads();

  // Prefix sums, written straight to global memory.
  const T tile_prefix = s_prefix;
#pragma unroll
  for (uint32_t r = 0; r < S::kRows; ++r) {
    uint4 q = vecs[first_vec + r * kWarp];
    T *qt = reinterpret_cast<T *>(&q);
    T x = tile_prefix + at[r];
#pragma unroll
    for (uint32_t e = 0; e < S::kPerVec; ++e) {
      const T v = qt[e];
      if (Inclusive) {
        x += v;
        qt[e] = x;
      } else {
        qt[e] = x;
        x += v;
      }
    }
    if (bulk) {
      reinterpret_cast<uint4 *>(data + base)[first_vec + r * kWarp] = q;
    } else {
      const uint64_t i0 = base + static_cast<uint64_t>(first_vec + r * kWarp) * S::kPerVec;
#pragma unroll
      for (uint32_t e = 0; e < S::kPerVec; ++e)
        if (i0 + e < count) data[i0 + e] = qt[e];
    }
  }
}

// Up to 64 KB of data: one block holds it in registers, with no records, so
// nothing is cleared first (a launch instead of a memset and a launch:
// 10,007 u32 8.4 -> 7.1 us of back-to-back calls on B200).
constexpr uint32_t kSmallBlock = 512, kSmallRows = 8;
template <class T> constexpr uint32_t small_max() {
  return kSmallBlock * kSmallRows * (16u / sizeof(T));
}

template <class T, bool Inclusive, bool Vectorised>
__global__ void __launch_bounds__(kSmallBlock)
    scan_small_kernel(T *__restrict__ data, uint32_t count, uint32_t *status) {
  constexpr uint32_t kPerVec = 16 / sizeof(T), kWarps = kSmallBlock / kWarp;
  __shared__ T s_warp[kWarps];
  const uint32_t t = threadIdx.x, lane = lane_id(), warp = t / kWarp;
  if (t == 0) *status = kDevOk;
  T v[kSmallRows][kPerVec], at[kSmallRows], run = 0;
  const uint32_t first = (warp * kSmallRows * kWarp + lane) * kPerVec;
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; ++r) {
    const uint32_t i = first + r * kWarp * kPerVec;
    if (Vectorised && i + kPerVec <= count) {
      const uint4 q = reinterpret_cast<const uint4 *>(data)[i / kPerVec];
      const T *qt = reinterpret_cast<const T *>(&q);
#pragma unroll
      for (uint32_t e = 0; e < kPerVec; ++e) v[r][e] = qt[e];
    } else {
#pragma unroll
      for (uint32_t e = 0; e < kPerVec; ++e) v[r][e] = i + e < count ? data[i + e] : T(0);
    }
  }
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; ++r) {
    T sum = 0;
#pragma unroll
    for (uint32_t e = 0; e < kPerVec; ++e) sum += v[r][e];
    const T inc = warp_inclusive_sum<T>(sum);
    at[r] = run + inc - sum;
    run += __shfl_sync(kFullMask, inc, kWarp - 1);
  }
  if (lane == 0) s_warp[warp] = run;
  __syncthreads();
  T before = 0;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; ++w)
    if (w < warp) before += s_warp[w];
#pragma unroll
  for (uint32_t r = 0; r < kSmallRows; ++r) {
    const uint32_t i = first + r * kWarp * kPerVec;
    T x = before + at[r];
    uint4 q;
    T *qt = reinterpret_cast<T *>(&q);
#pragma unroll
    for (uint32_t e = 0; e < kPerVec; ++e) {
      const T y = x + v[r][e];
      qt[e] = Inclusive ? y : x;
      x = y;
    }
    if (Vectorised && i + kPerVec <= count) {
      reinterpret_cast<uint4 *>(data)[i / kPerVec] = q;
    } else {
#pragma unroll
      for (uint32_t e = 0; e < kPerVec; ++e)
        if (i + e < count) data[i + e] = qt[e];
    }
  }
}

// Tiles for the element size and tile shape that need the most records (u64
// in the smallest, 8 KB, tile).
uint32_t max_tiles(uint32_t count) {
  return ceil_div(count, Tile8<uint64_t>::kTile) + 1;
}

// Clears the header and the records of the call's tiles (at `base`, the
// header's address) and launches the scan.
template <class T, bool Inclusive, bool Vectorised, class S>
vx_status launch_shape(T *data, uint32_t count, const ScanLayout &ws, cudaStream_t stream) {
  const uint32_t tiles = ceil_div(count, S::kTile);
  char *end = nullptr;
  const auto records = make_records<T>(ws, tiles, &end);
  char *base = reinterpret_cast<char *>(ws.tile_counter);
  VX_TRY_CUDA(cudaMemsetAsync(base, 0, static_cast<size_t>(end - base), stream));
  prof::Scope scope(sizeof(T) == 4 ? "scan_u32" : "scan_u64", stream);
  scan_kernel<T, Inclusive, Vectorised, S><<<tiles, S::kBlock, 0, stream>>>(data, count, ws,
                                                                            records);
  return from_cuda(cudaGetLastError());
}

// One block when the data fits it; else the tile shape of the "scan.tile_kb"
// knob (32, 16 or 8 KB tiles).
template <class T, bool Inclusive, bool Vectorised>
vx_status launch_tuned(T *data, uint32_t count, const ScanLayout &ws, cudaStream_t stream) {
  if (count <= small_max<T>()) {
    prof::Scope scope(sizeof(T) == 4 ? "scan_u32" : "scan_u64", stream);
    scan_small_kernel<T, Inclusive, Vectorised><<<1, kSmallBlock, 0, stream>>>(data, count,
                                                                               ws.status);
    return from_cuda(cudaGetLastError());
  }
  switch (tune::get(tune::kScanTileKb)) {
  case 8: return launch_shape<T, Inclusive, Vectorised, Tile8<T>>(data, count, ws, stream);
  case 16: return launch_shape<T, Inclusive, Vectorised, Tile16<T>>(data, count, ws, stream);
  default: return launch_shape<T, Inclusive, Vectorised, Tile32<T>>(data, count, ws, stream);
  }
}

} // namespace

size_t workspace_size(uint32_t count) {
  if (count == 0) return 0;
  const uint32_t tiles = max_tiles(count);
  Sizer s;
  s.take<uint32_t>(2);        // tile counter, status
  s.take<uint64_t>(tiles);    // packed records / u64 aggregates
  s.take<uint64_t>(tiles);    // u64 inclusive values
  s.take<uint32_t>(tiles);    // u64 record states
  return s.offset;
}

ScanLayout carve(void *workspace, uint32_t count) {
  const uint32_t tiles = max_tiles(count);
  Carver c(workspace);
  ScanLayout l;
  uint32_t *hdr = c.take<uint32_t>(2);
  l.tile_counter = hdr;
  l.status = hdr + 1;
  l.rec_a = c.take<uint64_t>(tiles);
  l.rec_b = c.take<uint64_t>(tiles);
  l.rec_state = c.take<uint32_t>(tiles);
  return l;
}

template <class T>
vx_status scan_launch(T *data, uint32_t count, bool inclusive, void *workspace,
                      size_t workspace_bytes, cudaStream_t stream) {
  if (data == nullptr && count != 0) return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  if (workspace == nullptr || workspace_bytes < workspace_size(count))
    return VX_ERR_INVALID_VALUE;
  const ScanLayout ws = carve(workspace, count);
  const bool vec = (reinterpret_cast<uintptr_t>(data) & 15u) == 0;
  if (inclusive)
    return vec ? launch_tuned<T, true, true>(data, count, ws, stream)
               : launch_tuned<T, true, false>(data, count, ws, stream);
  return vec ? launch_tuned<T, false, true>(data, count, ws, stream)
             : launch_tuned<T, false, false>(data, count, ws, stream);
}

template vx_status scan_launch<uint32_t>(uint32_t *, uint32_t, bool, void *,
                                         size_t, cudaStream_t);
template vx_status scan_launch<uint64_t>(uint64_t *, uint32_t, bool, void *,
                                         size_t, cudaStream_t);

} // namespace scan
} // namespace vx

extern "C" {

size_t vx_scan_workspace_size(uint32_t count) {
  return vx::scan::workspace_size(count);
}

vx_status vx_scan_exclusive_sum_u32(uint32_t *data, uint32_t count,
                                    void *workspace, size_t workspace_bytes,
                                    vx_stream stream) {
  return vx::scan::scan_launch<uint32_t>(data, count, false, workspace,
                                         workspace_bytes,
                                         static_cast<cudaStream_t>(stream));
}

vx_status vx_scan_inclusive_sum_u32(uint32_t *data, uint32_t count,
                                    void *workspace, size_t workspace_bytes,
                                    vx_stream stream) {
  return vx::scan::scan_launch<uint32_t>(data, count, true, workspace,
                                         workspace_bytes,
                                         static_cast<cudaStream_t>(stream));
}

vx_status vx_scan_exclusive_sum_u64(uint64_t *data, uint32_t count,
                                    void *workspace, size_t workspace_bytes,
                                    vx_stream stream) {
  return vx::scan::scan_launch<uint64_t>(data, count, false, workspace,
                                         workspace_bytes,
                                         static_cast<cudaStream_t>(stream));
}

} // extern "C"

// ------------------------------------------------- allocation-free variant --
//
// Some callers cannot allocate device memory at the point where they need a
// prefix sum: a frame loop or plugin that owns a fixed device-memory budget,
// or code that must not call cudaMalloc / cudaFree because those calls
// synchronise the device.  This entry point takes no workspace: its look-back
// scratch is one array in this library's own device memory, sized for at
// most kNoAllocMaxCount elements (272 KiB plus a 256-byte header, held on
// every GPU that loads the library until the process exits).

namespace vx::scan {
namespace {

constexpr uint32_t kNoAllocMaxCount = 1u << 28;
constexpr uint32_t kNoAllocTiles =
    (kNoAllocMaxCount + Tile32<uint32_t>::kTile - 1) / Tile32<uint32_t>::kTile;
constexpr uint32_t kNoAllocRecords = kNoAllocTiles + 2 * ((kNoAllocTiles + kGroup - 1) / kGroup);
constexpr size_t kNoAllocHeader = 256; // tile counter, status word

// [0, 256): tile counter and status; then a look-back record per tile and two
// words per group of tiles.
static __device__ __align__(256) unsigned char
    g_noalloc_scratch[kNoAllocHeader + size_t(kNoAllocRecords) * sizeof(uint64_t)];

// Unique id of the calling thread's current CUDA context (0 when there is
// none or the driver entry points are unavailable).  Context ids are never
// reused within a process, so a context created again after a device reset
// gets a new id even when its handle value repeats.
unsigned long long current_context_id() {
  using GetCurrent = CUresult (*)(CUcontext *);
  using GetId = CUresult (*)(CUcontext, unsigned long long *);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f);
  });
  if (get_current == nullptr || get_id == nullptr) return 0;
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return 0;
  if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Device address of g_noalloc_scratch in the current context (the symbol's
// name is only a host-side stand-in and must never be handed to a kernel).
// The address is looked up with cudaGetSymbolAddress once per context and
// cached under the context's unique id, so a device reset (which unloads the
// module) is followed by a fresh lookup instead of a dangling address.  When
// the context id cannot be read, the address is looked up on every call.
void *noalloc_scratch(cudaError_t *err) {
  static std::mutex mu;
  static unsigned long long cached_ctx = 0;
  static void *cached_addr = nullptr;
  *err = cudaSuccess;
  unsigned long long ctx = current_context_id();
  std::lock_guard<std::mutex> lock(mu);
  if (ctx != 0 && ctx == cached_ctx && cached_addr != nullptr) return cached_addr;
  void *p = nullptr;
  *err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (*err != cudaSuccess) return nullptr;
  if (ctx == 0) ctx = current_context_id(); // the lookup may have created the context
  cached_ctx = ctx;
  cached_addr = ctx != 0 ? p : nullptr;
  return p;
}

} // namespace
} // namespace vx::scan

extern "C" {

// Allocation-free exclusive sum (see the block comment above): count must be
// at most 2^28; every call on a device shares one scratch array, so calls that
// may overlap on the GPU (different streams without ordering) race.  The
// first call in each CUDA context looks the scratch address up and should
// come before any stream capture; vx_scan_noalloc_status reads the status
// word this call leaves behind.
vx_status vx_scan_exclusive_sum_u32_noalloc(uint32_t *data, uint32_t count,
                                            vx_stream stream) {
  using namespace vx::scan;
  if (data == nullptr && count != 0) return VX_ERR_INVALID_VALUE;
  if (count > kNoAllocMaxCount) return VX_ERR_CAPACITY;
  if (count == 0) return VX_OK;
  cudaError_t err = cudaSuccess;
  char *base = static_cast<char *>(noalloc_scratch(&err));
  if (base == nullptr) return vx::from_cuda(err);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  ScanLayout ws{};
  ws.tile_counter = reinterpret_cast<uint32_t *>(base);
  ws.status = ws.tile_counter + 1;
  ws.rec_a = reinterpret_cast<uint64_t *>(base + kNoAllocHeader);
  if ((reinterpret_cast<uintptr_t>(data) & 15u) == 0)
    return launch_shape<uint32_t, false, true, Tile32<uint32_t>>(data, count, ws, s);
  return launch_shape<uint32_t, false, false, Tile32<uint32_t>>(data, count, ws, s);
}

// Status of the most recent allocation-free scan on the current device:
// synchronises the stream, then reads the device status word that the scan
// kernel leaves in the shared scratch (VX_ERR_TIMEOUT when a look-back wait
// gave up, in which case that call's prefix sums are not valid).  Every call
// of the allocation-free scan clears the word first, so this reports the last
// call that ran before the read; with calls that overlap on the GPU the word
// belongs to whichever wrote it last.
vx_status vx_scan_noalloc_status(vx_stream stream) {
  using namespace vx::scan;
  cudaError_t err = cudaSuccess;
  char *base = static_cast<char *>(noalloc_scratch(&err));
  if (base == nullptr) return vx::from_cuda(err);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint32_t code = 0;
  VX_TRY_CUDA(cudaMemcpyAsync(&code, base + sizeof(uint32_t), sizeof(code),
                              cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  return vx::status_from_device(code);
}

} // extern "C"
