// Shared pieces of the batched edit pipelines (Hash DAG and SVO).
//
// Both structures are edited by the same top-down, level-synchronous
// expansion.  A work item is one octree cell that at least one primitive
// touches but does not decide completely.  It carries the cell, the ref of the
// structure that was there before (or a uniform constant), and the ordered
// list of primitive indices that still matter inside it.  For each of its 8
// children the expansion finds the last primitive that covers the child
// entirely: every earlier primitive is overwritten there, so the child starts
// from that primitive's uniform value, and only later primitives that cut the
// child partially travel down.  Children that no primitive touches keep their
// old subtree (copy-on-write).  The result is exactly sequential application
// of the primitives in array order.
#pragma once

#include "common.cuh"
#include "voxel_b200_device.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace vx::edit {

// Internal primitive shapes beyond the public sphere / box.
constexpr uint32_t kShapeLeafMask = 2; // c = leaf origin, r[0..1] = mask lo/hi
constexpr uint32_t kShapeTerrain = 3;  // c = {seed, scale, caves}

constexpr uint32_t kBlock = 256;

struct Cell {
  uint32_t x, y, z; // cell index at its level
};

__host__ __device__ __forceinline__ uint64_t pack_cell(uint32_t x, uint32_t y,
                                                       uint32_t z) {
  return static_cast<uint64_t>(x) | (static_cast<uint64_t>(y) << 21) |
         (static_cast<uint64_t>(z) << 42);
}
__host__ __device__ __forceinline__ Cell unpack_cell(uint64_t p) {
  return Cell{static_cast<uint32_t>(p & 0x1fffff),
              static_cast<uint32_t>((p >> 21) & 0x1fffff),
              static_cast<uint32_t>((p >> 42) & 0x1fffff)};
}
__host__ __device__ __forceinline__ uint64_t child_cell(uint64_t p, uint32_t c) {
  const Cell k = unpack_cell(p);
  return pack_cell(2 * k.x + (c & 1u), 2 * k.y + ((c >> 1) & 1u),
                   2 * k.z + ((c >> 2) & 1u));
}

// Exact sphere tests in 32-bit arithmetic for radii below 2^14: a distance
// that decides anything is at most r (+3 inside a leaf), so every square and
// every sum of three squares stays below 2^31.  Larger radii take the 64-bit
// definitions of vx_workload.h; both give identical results.
constexpr int64_t kFastRadius = int64_t(1) << 14;

// Cells lie in [0, 2^16] per axis (depth <= 14); a centre clamped to
// [-2^16, 2^18] keeps every outcome (a clamped centre is still more than
// 2^14 > r away from every cell), so the differences fit in 32 bits.
__device__ __forceinline__ uint32_t sphere_classify32(const vx_primitive &p, int64_t ox,
                                                      int64_t oy, int64_t oz, int64_t n) {
  const int32_t r = static_cast<int32_t>(p.r[0]);
  const int32_t lo[3] = {static_cast<int32_t>(ox), static_cast<int32_t>(oy),
                         static_cast<int32_t>(oz)};
  const int32_t n1 = static_cast<int32_t>(n) - 1;
  uint32_t near2 = 0, far2 = 0;
  bool far_in = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int32_t c = max(-(1 << 16), min(1 << 18, p.c[a]));
    const int32_t a0 = lo[a], a1 = lo[a] + n1;
    const int32_t d = c < a0 ? a0 - c : (c > a1 ? c - a1 : 0);
    if (d > r) return VX_CELL_EMPTY;
    near2 += static_cast<uint32_t>(d) * static_cast<uint32_t>(d);
    const int32_t f = max(abs(c - a0), abs(c - a1));
    if (f > r) far_in = false;
    else far2 += static_cast<uint32_t>(f) * static_cast<uint32_t>(f);
  }
  const uint32_t r2 = static_cast<uint32_t>(r) * static_cast<uint32_t>(r);
  if (near2 > r2) return VX_CELL_EMPTY;
  return (far_in && far2 <= r2) ? VX_CELL_FULL : VX_CELL_MIXED;
}

// Sphere mask of the leaf at o; the caller has classified the leaf MIXED, so
// every coordinate difference is within r + 3 of the centre.
__device__ __forceinline__ uint64_t sphere_leaf_mask32(const vx_primitive &p, int64_t ox,
                                                       int64_t oy, int64_t oz) {
  const int32_t r = static_cast<int32_t>(p.r[0]);
  const int32_t r2 = r * r;
  const int32_t dx0 = static_cast<int32_t>(ox - p.c[0]);
  const int32_t dy0 = static_cast<int32_t>(oy - p.c[1]);
  const int32_t dz0 = static_cast<int32_t>(oz - p.c[2]);
  int32_t dx2[4], dy2[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    dx2[i] = (dx0 + i) * (dx0 + i);
    dy2[i] = (dy0 + i) * (dy0 + i);
  }
  uint64_t m = 0;
#pragma unroll
  for (int z = 0; z < 4; ++z) {
    const int32_t rz = r2 - (dz0 + z) * (dz0 + z);
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int32_t ry = rz - dy2[y];
      const uint32_t bits = (dx2[0] <= ry ? 1u : 0u) | (dx2[1] <= ry ? 2u : 0u) |
                            (dx2[2] <= ry ? 4u : 0u) | (dx2[3] <= ry ? 8u : 0u);
      m |= static_cast<uint64_t>(ry >= 0 ? bits : 0u) << (4 * y + 16 * z);
    }
  }
  return m;
}

// The same mask for radii up to kFloatMaskRadius, in single precision: the
// caller has classified the leaf MIXED, so every coordinate difference is at
// most r + 3 and every value below is an integer under 2^22 in magnitude,
// which each single-precision operation (contracted or not) keeps exact.  A
// voxel is inside when sx <= r^2 - sy - sz, i.e. when sx - (r^2 + 1 - sy -
// sz) is negative; an exact zero is +0, so the sign bit is the voxel's bit.
// The sign bits are shifted into the mask one funnel shift per voxel, the
// highest voxel first: a subtraction and a shift per voxel.
constexpr uint32_t kFloatMaskRadius = 1024;

// (fx, fy, fz): the leaf's first voxel relative to the centre; r2p1 = r^2 + 1.
__device__ __forceinline__ uint64_t sphere_mask_rows(float fx, float fy, float fz, float r2p1) {
  float sx[4], sy[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = fx + static_cast<float>(i), b = fy + static_cast<float>(i);
    sx[i] = a * a;
    sy[i] = b * b;
  }
  uint32_t half[2] = {0u, 0u};
#pragma unroll
  for (int z = 3; z >= 0; --z) {
    const float c = fz + static_cast<float>(z);
    const float tz = r2p1 - c * c;
#pragma unroll
    for (int y = 3; y >= 0; --y) {
      const float t = tz - sy[y];
#pragma unroll
      for (int i = 3; i >= 0; --i)
        half[z >> 1] = __funnelshift_l(__float_as_uint(sx[i] - t), half[z >> 1], 1);
    }
  }
  return (static_cast<uint64_t>(half[1]) << 32) | half[0];
}

__device__ __forceinline__ uint64_t sphere_leaf_mask_f32(const vx_primitive &p, int64_t ox,
                                                        int64_t oy, int64_t oz) {
  const float r = static_cast<float>(p.r[0]);
  return sphere_mask_rows(static_cast<float>(static_cast<int32_t>(ox - p.c[0])),
                          static_cast<float>(static_cast<int32_t>(oy - p.c[1])),
                          static_cast<float>(static_cast<int32_t>(oz - p.c[2])), r * r + 1.0f);
}

// Children (side n, one bit each) of the cell at o that a sphere of radius
// below kFastRadius touches and covers: the nearest and farthest squared
// distances per axis are found once for each half of the cell and summed per
// child (sphere_classify32 child by child costs four times the
// instructions).  Distances are clamped to r + 1, which keeps every square
// and sum below 2^31 and every outcome.
__device__ __forceinline__ void sphere_classify_children(const vx_primitive &p, uint32_t ox,
                                                         uint32_t oy, uint32_t oz, uint32_t n,
                                                         uint32_t &touched, uint32_t &covered) {
  const int32_t r = static_cast<int32_t>(p.r[0]), side = static_cast<int32_t>(n);
  const int32_t lo[3] = {static_cast<int32_t>(ox), static_cast<int32_t>(oy),
                         static_cast<int32_t>(oz)};
  int32_t near2[3][2], far2[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int32_t c = max(-(1 << 16), min(1 << 18, p.c[a]));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int32_t a0 = lo[a] + side * h, a1 = a0 + side - 1;
      const int32_t d = min(max(max(a0 - c, c - a1), 0), r + 1);
      const int32_t f = min(max(c - a0, a1 - c), r + 1); // the farther end
      near2[a][h] = d * d;
      far2[a][h] = f * f;
    }
  }
  const int32_t r2 = r * r;
  touched = covered = 0;
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    const int32_t d = near2[0][c & 1u] + near2[1][(c >> 1) & 1u] + near2[2][c >> 2];
    const int32_t f = far2[0][c & 1u] + far2[1][(c >> 1) & 1u] + far2[2][c >> 2];
    if (d <= r2) touched |= 1u << c;
    if (f <= r2) covered |= 1u << c;
  }
}

// Classify primitive p against the voxel cube [o, o + n)^3.  Kernels that
// only ever see sphere / box / leaf-mask primitives instantiate Terrain =
// false and carry none of the terrain generator's code.
template <bool Terrain>
__device__ __forceinline__ uint32_t classify(const vx_primitive &p,
                                             uint32_t world_exp, int64_t ox,
                                             int64_t oy, int64_t oz, int64_t n) {
  const uint32_t shape = vx_prim_shape(&p);
  if (Terrain && shape == kShapeTerrain) {
    const vx_terrain t{static_cast<uint32_t>(p.c[0]), static_cast<uint32_t>(p.c[1]),
                       static_cast<uint32_t>(p.c[2]), world_exp};
    return vx_terrain_classify(&t, static_cast<uint32_t>(ox),
                               static_cast<uint32_t>(oy),
                               static_cast<uint32_t>(oz), static_cast<uint32_t>(n));
  }
  if (shape == kShapeLeafMask) {
    const int64_t lx = p.c[0], ly = p.c[1], lz = p.c[2];
    if (lx < ox || lx >= ox + n || ly < oy || ly >= oy + n || lz < oz ||
        lz >= oz + n)
      return VX_CELL_EMPTY;
    return VX_CELL_MIXED;
  }
  if (shape == VX_SHAPE_SPHERE && p.r[0] < kFastRadius)
    return sphere_classify32(p, ox, oy, oz, n);
  return vx_prim_classify(&p, ox, oy, oz, n);
}

// Voxels of the 4^3 leaf at o that the primitive covers.
template <bool Terrain>
__device__ __forceinline__ uint64_t leaf_mask(const vx_primitive &p,
                                              uint32_t world_exp, int64_t ox,
                                              int64_t oy, int64_t oz) {
  const uint32_t shape = vx_prim_shape(&p);
  if (Terrain && shape == kShapeTerrain) {
    const vx_terrain t{static_cast<uint32_t>(p.c[0]), static_cast<uint32_t>(p.c[1]),
                       static_cast<uint32_t>(p.c[2]), world_exp};
    return vx_terrain_leaf_mask(&t, static_cast<uint32_t>(ox),
                                static_cast<uint32_t>(oy), static_cast<uint32_t>(oz));
  }
  if (shape == kShapeLeafMask) {
    if (p.c[0] != ox || p.c[1] != oy || p.c[2] != oz) return 0;
    return static_cast<uint64_t>(p.r[0]) | (static_cast<uint64_t>(p.r[1]) << 32);
  }
  if (shape == VX_SHAPE_SPHERE && p.r[0] <= kFloatMaskRadius)
    return sphere_leaf_mask_f32(p, ox, oy, oz);
  if (shape == VX_SHAPE_SPHERE && p.r[0] < kFastRadius)
    return sphere_leaf_mask32(p, ox, oy, oz);
  return vx_prim_leaf_mask(&p, ox, oy, oz);
}

// Children of the packed cell `cell` (side n each) that any edit primitive
// touches (bits 0-7) and covers (bits 8-15); a function of its own, so that
// its registers do not weigh on the loops that mostly meet spheres.
static __device__ __noinline__ uint32_t other_children(const vx_primitive *prim, uint64_t cell,
                                                       uint32_t n) {
  const vx_primitive p = *prim;
  const uint32_t shape = vx_prim_shape(&p);
  const int64_t o[3] = {static_cast<int64_t>(cell & 0x1fffff) * 2 * n,
                        static_cast<int64_t>((cell >> 21) & 0x1fffff) * 2 * n,
                        static_cast<int64_t>((cell >> 42) & 0x1fffff) * 2 * n};
  uint32_t touched = 0, covered = 0;
  if (shape == VX_SHAPE_SPHERE || shape == kShapeLeafMask) {
    for (uint32_t c = 0; c < 8; ++c) {
      const uint32_t cls = classify<false>(p, 0, o[0] + (c & 1u) * n, o[1] + ((c >> 1) & 1u) * n,
                                           o[2] + (c >> 2) * n, n);
      if (cls != VX_CELL_EMPTY) touched |= 1u << c;
      if (cls == VX_CELL_FULL) covered |= 1u << c;
    }
  } else { // boxes: per axis and half, then all children
    uint32_t meets[3] = {0, 0, 0}, inside[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      int64_t b0, b1;
      vx_prim_axis_range(&p, a, &b0, &b1);
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const int64_t a0 = o[a] + h * n, a1 = a0 + n - 1;
        if (b1 >= a0 && b0 <= a1) meets[a] |= 1u << h;
        if (b0 <= a0 && b1 >= a1) inside[a] |= 1u << h;
      }
    }
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      touched |= ((meets[0] >> (c & 1u)) & (meets[1] >> ((c >> 1) & 1u)) & (meets[2] >> (c >> 2)) & 1u) << c;
      covered |= ((inside[0] >> (c & 1u)) & (inside[1] >> ((c >> 1) & 1u)) & (inside[2] >> (c >> 2)) & 1u) << c;
    }
  }
  return touched | (covered << 8);
}

// The voxels of leaf c of the 8^3 cell `cell` that any edit primitive covers
// (a function of its own for the same reason).
static __device__ __noinline__ uint64_t other_leaf_mask(const vx_primitive *prim, uint64_t cell,
                                                        uint32_t c) {
  const vx_primitive p = *prim;
  const Cell k = unpack_cell(cell);
  const int64_t ox = int64_t(2 * k.x + (c & 1u)) * 4;
  const int64_t oy = int64_t(2 * k.y + ((c >> 1) & 1u)) * 4;
  const int64_t oz = int64_t(2 * k.z + (c >> 2)) * 4;
  const uint32_t cls = classify<false>(p, 0, ox, oy, oz, 4);
  if (cls == VX_CELL_EMPTY) return 0ull;
  return cls == VX_CELL_FULL ? ~0ull : leaf_mask<false>(p, 0, ox, oy, oz);
}

// One work item of the top-down expansion (32 bytes).  Two fields change
// meaning over an edit: `pstart`, once the item is expanded, counts its child
// items that have not finished yet, and `result`, until the item is rebuilt,
// holds its parent's item index (kNoParent for the root), so that a
// bottom-up build can run without level barriers: the last child to finish
// rebuilds its parent.
struct Item {
  uint64_t cell;
  uint32_t old;        // ref (DAG) or slot word (SVO) of the previous content
  uint32_t pstart;     // first pair of this item in its level's pair array; then pending children
  uint32_t pcount;     // number of pairs
  uint32_t child_base; // first child item at the next level
  uint32_t masks;      // child_mask | const_mask << 8 | const_full << 16
  uint32_t result;     // parent index until rebuilt, then the rebuilt ref / slot word
};
constexpr uint32_t kNoParent = 0xffffffffu;

// Item reads on a climb (another SM wrote the item or its children's
// results in this launch): from L2, never from this SM's L1.
__device__ __forceinline__ Item load_item_l2(const Item *p) {
  const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(p));
  const uint4 b = __ldcg(reinterpret_cast<const uint4 *>(p) + 1);
  Item it;
  it.cell = static_cast<uint64_t>(a.x) | (static_cast<uint64_t>(a.y) << 32);
  it.old = a.z;
  it.pstart = a.w;
  it.pcount = b.x;
  it.child_base = b.y;
  it.masks = b.z;
  it.result = b.w;
  return it;
}
static_assert(sizeof(Item) == 32, "Item is 32 bytes");

// Per-edit device bookkeeping (one per structure).
struct Header {
  uint32_t root;
  uint32_t status;
  uint32_t prim_count;          // primitives of the current submission
  uint32_t pad0;
  uint32_t item_off[16];        // first item of each level
  uint32_t item_count[16];      // items of each level
  uint32_t pair_count[16];      // pairs of each level
  uint64_t node_count[16];      // items inserted per table (DAG)
  uint32_t pool_used[16];       // words used per level pool (DAG)
  uint32_t big_count[16];       // items with long lists (EditCtx::big_item)
  uint32_t pool_mark[16];       // pool_used before this edit's inserts (DAG)
};

struct Arena {
  Item *items;
  uint32_t *pairs[2];
  uint32_t *big;       // indices of items with long primitive lists
  uint32_t item_cap;
  uint32_t pair_cap;
  uint32_t big_cap;
};

// Items with more primitives than EditCtx::big_item (the tuning knob
// "edit.big_item", 32 by default) are expanded apart: in batches by
// expand_long_kernel (a cluster of eight blocks above 4,096 primitives, a block
// below), in small edits by a block (expand_big_body).  They are listed when
// they are emitted (the level above's expansion, or the init of
// the root), so that a level's short and long lists can be expanded side by
// side; the big buffer's two halves alternate by level, so level l + 1's
// list fills while level l's is read.
__device__ __forceinline__ uint32_t *big_list(const Arena &a, uint32_t l) {
  return a.big + (l & 1u) * (a.big_cap / 2u);
}


// init_kernel's root_old value meaning "the root stored in the header".
constexpr uint32_t kUseHeaderRoot = 0xfffffffeu;

// Device-side edit context shared by the DAG and SVO pipelines.
struct EditCtx {
  Header *hdr;
  Arena a;
  const vx_primitive *prims;
  const uint32_t *d_prim_count; // device count (NULL: use host_prim_count)
  uint32_t host_prim_count;
  uint32_t depth;
  uint32_t big_item; // items with longer primitive lists are listed (big_list)
  // Not NULL: the primitives are leaf masks of distinct leaves in ascending
  // leaf key (Morton) order, with these keys, so an item's list is a range of
  // them (expand_sorted_body).
  const uint64_t *sorted_keys;
};

// List item `idx` of level l (its index within the level) for the
// long lists' expansion when its primitive list is long and level l is
// expanded at all (levels below depth - 1).
__device__ __forceinline__ void note_big(const EditCtx &x, uint32_t l, uint32_t idx,
                                         uint32_t pcount) {
  if (pcount <= x.big_item || l + 1 >= x.depth) return;
  const uint32_t slot = atomicAdd(&x.hdr->big_count[l], 1u);
  if (slot < x.a.big_cap / 2u) big_list(x.a, l)[slot] = idx;
  else set_status(&x.hdr->status, kDevCapacity);
}

// A tree Policy supplies:
//   static constexpr bool kItemsForConst  - also create a (primitive-free)
//       child item where a primitive covers the child entirely, so the
//       rebuild sees its constant value in the child item's `old`;
//   child(l, old, c)                      - content of child c of `old` at level l;
//   children(l, old, ref)                 - all eight of them;
//   classify<Terrain>(prim, world_exp, ox, oy, oz, n);
//   const_value(prim, oz, n)              - the content a fully covering
//       primitive leaves in the cube at height oz of side n (1 = full);
//   static constexpr uint32_t kValueBits  - the bits of an edit primitive's
//       flags that decide it;
//   replaced(l, old, c)                   - child c of `old` is overwritten
//       by a fully covering primitive (its subtree is dropped).

// The blocks a pipeline stage runs on: its own launch (blockIdx / gridDim), or
// the whole grid of the single cooperative kernel that runs every stage of a
// small edit in a row.
struct Blocks {
  uint32_t id, count;
};
__device__ __forceinline__ Blocks launch_blocks() { return Blocks{blockIdx.x, gridDim.x}; }

// True on every thread of the block when the edit's status is no longer ok.
// Block-uniform, so a stage that returns on it never leaves part of a block
// at a barrier.
__device__ __forceinline__ bool edit_failed(const Header *h) {
  return __syncthreads_or(ld_relaxed_u32(&h->status) != kDevOk) != 0;
}

__device__ __forceinline__ void init_body(EditCtx x, uint32_t root_old, Blocks blk) {
  Header *h = x.hdr;
  // With a device-side count, host_prim_count is the capacity of the list.
  const uint32_t dn = x.d_prim_count ? *x.d_prim_count : 0u;
  if (x.d_prim_count && dn > x.host_prim_count) {
    if (blk.id == 0 && threadIdx.x == 0) set_status(&h->status, kDevInvalid);
    return;
  }
  const uint32_t n = x.d_prim_count ? dn : x.host_prim_count;
  if (blk.id == 0 && threadIdx.x == 0) {
    for (uint32_t l = 0; l < 16; ++l) {
      h->item_off[l] = 0;
      h->item_count[l] = 0;
      h->pair_count[l] = 0;
      h->big_count[l] = 0;
    }
    h->prim_count = n;
    const uint32_t ok = h->status == kDevOk && n <= x.a.pair_cap;
    if (h->status == kDevOk && n > x.a.pair_cap) h->status = kDevCapacity;
    if (ok) {
      h->item_count[0] = 1;
      h->pair_count[0] = n;
      Item it{};
      it.cell = 0;
      it.old = root_old == kUseHeaderRoot ? h->root : root_old;
      it.pstart = 0;
      it.pcount = n;
      it.result = kNoParent;
      x.a.items[0] = it;
      note_big(x, 0, 0, n);
    }
  }
  if (n > x.a.pair_cap) return;
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
       i < n; i += static_cast<uint64_t>(blk.count) * blockDim.x) {
    x.a.pairs[0][i] = static_cast<uint32_t>(i);
    if (x.sorted_keys != nullptr) x.a.pairs[1][i] = static_cast<uint32_t>(i);
  }
}

static __global__ void init_kernel(EditCtx x, uint32_t root_old) {
  init_body(x, root_old, launch_blocks());
}

// ------------------------------------------- plain voxel lists, small edits --
//
// Inside the single cooperative kernel of a small edit, a voxel list (one op
// for every voxel) becomes its leaf-mask primitives without a sort: voxels
// are aggregated into a hash table of {leaf key + 1, mask} slots (atomicCAS
// claims a slot and lists it, atomicOr sets the voxel's bit), then primitive
// i is written from the i-th listed slot.  One op for all voxels makes the
// order of the primitives irrelevant.  Stages: clear, aggregate, fill (the
// last beside the edit's init, which only needs the count), each followed by
// a grid-wide barrier.
struct PlainPrep {
  const vx_voxel *edits;
  uint32_t count;       // voxels
  uint32_t op, material;
  ulonglong2 *slots;    // {packed leaf coordinates + 1 (0 = free), mask}
  uint32_t nslots;
  uint32_t *order;      // used slots in the order they were claimed
  vx_primitive *prims;  // out: one leaf-mask primitive per touched leaf
  uint32_t *nprims;     // out: their number (the edit's device-side count)
};

// The prep's table and primitive list carved from a plain-path workspace;
// false when they do not fit it.
inline bool plain_prep_layout(void *ws, size_t ws_bytes, const vx_voxel *edits, uint32_t count,
                              uint32_t op, uint32_t material, PlainPrep *out) {
  Carver c(ws);
  PlainPrep p{};
  p.edits = edits;
  p.count = count;
  p.op = op;
  p.material = material;
  p.nslots = count + count / 2u + 1u; // distinct leaves <= count: load <= 2/3
  p.slots = c.take<ulonglong2>(p.nslots);
  p.order = c.take<uint32_t>(count);
  p.prims = c.take<vx_primitive>(count);
  p.nprims = c.take<uint32_t>(1);
  if (c.offset > ws_bytes) return false;
  *out = p;
  return true;
}

__device__ __forceinline__ void plain_prep_clear(const PlainPrep &p, Blocks blk) {
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < p.nslots;
       i += static_cast<uint64_t>(blk.count) * blockDim.x)
    p.slots[i] = make_ulonglong2(0ull, 0ull);
  if (blk.id == 0 && threadIdx.x == 0) *p.nprims = 0;
}

__device__ __forceinline__ void plain_prep_aggregate(const PlainPrep &p, uint32_t depth,
                                                     Blocks blk) {
  const uint32_t side_exp = depth + 2;
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < p.count;
       i += static_cast<uint64_t>(blk.count) * blockDim.x) {
    const vx_voxel v = p.edits[i];
    if ((v.x >> side_exp) | (v.y >> side_exp) | (v.z >> side_exp)) continue; // outside: ignored
    const uint64_t key = (static_cast<uint64_t>(v.x >> 2) | (static_cast<uint64_t>(v.y >> 2) << 21) |
                          (static_cast<uint64_t>(v.z >> 2) << 42)) + 1ull;
    const uint64_t bit = 1ull << ((v.x & 3u) + 4u * (v.y & 3u) + 16u * (v.z & 3u));
    uint32_t pos = vx_reduce_hash(vx_mix64(key), p.nslots);
    for (uint32_t probe = 0; probe < p.nslots; ++probe) {
      const unsigned long long old =
          atomicCAS(reinterpret_cast<unsigned long long *>(&p.slots[pos].x), 0ull, key);
      if (old == 0ull || old == key) {
        if (old == 0ull) p.order[atomicAdd(p.nprims, 1u)] = pos; // distinct leaves <= count
        atomicOr(reinterpret_cast<unsigned long long *>(&p.slots[pos].y), bit);
        break;
      }
      pos = pos + 1u == p.nslots ? 0u : pos + 1u;
    }
  }
}

__device__ __forceinline__ void plain_prep_fill(const PlainPrep &p, Blocks blk) {
  const uint32_t n = *p.nprims;
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(blk.count) * blockDim.x) {
    const ulonglong2 e = p.slots[p.order[i]];
    const uint64_t k = e.x - 1ull;
    vx_primitive pr{};
    pr.c[0] = static_cast<int32_t>((k & 0x1fffffull) * 4u);
    pr.c[1] = static_cast<int32_t>(((k >> 21) & 0x1fffffull) * 4u);
    pr.c[2] = static_cast<int32_t>(((k >> 42) & 0x1fffffull) * 4u);
    pr.r[0] = static_cast<uint32_t>(e.y);
    pr.r[1] = static_cast<uint32_t>(e.y >> 32);
    pr.flags = vx_make_flags(kShapeLeafMask, p.op, p.material);
    p.prims[i] = pr;
  }
}

// The value that a child's remaining primitives leave in the voxels they
// cover (full, empty or, with materials, one material), while it is the same
// for all.  When the child holds that value everywhere already (added to solid
// ground, removed from air), nothing below it changes: the child is left
// alone and no item goes down.  Half of the items of a sphere batch on
// terrain are of that kind (24.8 -> 12.6 M leaf-parent items at 16,384
// spheres in 16384^3).
// Kept as the flag bits that decide the value (operation, material), so that
// a primitive costs one comparison and the value is found once at the end.
template <class Policy> struct LeftValue {
  uint32_t bits = 0;
  bool same = true;
  __device__ __forceinline__ void add(const vx_primitive &p, bool first) {
    const uint32_t b = p.flags & Policy::kValueBits;
    same = first || (same && b == bits);
    bits = first ? b : bits;
  }
  __device__ __forceinline__ bool all(const Policy &pol, uint32_t held) const {
    vx_primitive p{};
    p.flags = bits;
    return same && pol.const_value(p, 0, 4) == held;
  }
};

// Top-down expansion of level l into level l + 1 (l + 1 < depth).  Eight
// lanes per work item, one per child cell: lane c walks the item's ordered
// primitive list once, remembering the last primitive that covers child c
// entirely (which resets the count of partial ones before it) and counting the
// partial ones after it; a second walk writes those to the child's list.
// Output space for a block's 32 items is taken with one atomicAdd per counter.
template <class Policy, bool Terrain>
__device__ __forceinline__ void expand_body(EditCtx x, Policy pol, uint32_t l, Blocks blk) {
  Header *h = x.hdr;
  // the level's counts load beside the status (one round trip, not two)
  const uint32_t W = h->item_count[l];
  const uint32_t base = h->item_off[l];
  if (edit_failed(h)) return;
  const uint32_t depth = x.depth;
  const uint32_t next_base = base + W;
  if (blk.id == 0 && threadIdx.x == 0) h->item_off[l + 1] = next_base;
  const uint32_t *in_pairs = x.a.pairs[l & 1u];
  uint32_t *out_pairs = x.a.pairs[(l + 1) & 1u];
  const int64_t csize = int64_t(4) << (depth - l - 1); // child cell size
  const uint32_t world_exp = depth + 2;
  constexpr uint32_t kGroups = kBlock / 8;
  static_assert(kGroups == kWarp, "one warp scans the groups' counts");

  __shared__ uint32_t s_items[kGroups], s_pairs[kGroups];
  __shared__ uint32_t s_item_base, s_pair_base;
  __shared__ bool s_room;
  // the group's current chunk of its item's list: pair values and primitives
  __shared__ uint32_t s_pidx[kGroups][8];
  __shared__ vx_primitive s_prim[kGroups][8];
  const uint32_t group = threadIdx.x >> 3, c = threadIdx.x & 7u;
  const uint32_t gshift = (lane_id() >> 3) * 8u; // this group's byte in a ballot
  const uint32_t gmask = 0xffu << gshift;        // this group's lanes

  for (uint64_t tile = blk.id; tile * kGroups < W; tile += blk.count) {
    const uint32_t wi = static_cast<uint32_t>(tile * kGroups) + group;
    const bool have = wi < W;
    Item it{};
    if (have) it = x.a.items[base + wi];
    // Items with long lists were listed when they were emitted (big_list).
    const bool big = have && it.pcount > x.big_item;
    if (big) it.pcount = 0;
    const Cell cell = unpack_cell(it.cell);
    const int64_t ox = int64_t(2 * cell.x + (c & 1u)) * csize;
    const int64_t oy = int64_t(2 * cell.y + ((c >> 1) & 1u)) * csize;
    const int64_t oz = int64_t(2 * cell.z + ((c >> 2) & 1u)) * csize;
    // The child's previous content, read before the list walk so that the
    // two chains of loads overlap (unused when a primitive covers the child).
    const uint32_t old_child = have && !big ? pol.child(l, it.old, c) : 0u;
    int32_t last_full = -1;
    uint32_t cnt = 0;
    // Bit k: the list's k-th primitive cuts this child partially and comes
    // after every primitive that covers it (kept for lists of up to 32).
    uint32_t partial = 0;
    // What those primitives leave in the voxels they cover, when all leave
    // the same: a child that holds just that everywhere needs no edit.
    LeftValue<Policy> left;
    // Eight primitives at a time: each lane of the group loads one pair and
    // its primitive (two rounds of independent loads per chunk instead of two
    // dependent loads per primitive), then every lane walks the chunk for its
    // own child.  pcount is the same on the group's lanes, so they pass the
    // group barriers together.
    // (A terrain build's items hold its one primitive: walked in place.)
    for (uint32_t k = 0; Terrain && k < it.pcount; ++k) {
      const uint32_t p = in_pairs[it.pstart + k];
      const uint32_t cls = pol.template classify<Terrain>(x.prims[p], world_exp, ox, oy, oz, csize);
      if (cls == VX_CELL_FULL) {
        last_full = static_cast<int32_t>(p);
        cnt = 0;
        partial = 0;
      } else if (cls == VX_CELL_MIXED) {
        ++cnt;
        if (k < 32u) partial |= 1u << k;
      }
    }
    for (uint32_t k0 = 0; !Terrain && k0 < it.pcount; k0 += 8) {
      if (k0 + c < it.pcount) {
        const uint32_t p = in_pairs[it.pstart + k0 + c];
        s_pidx[group][c] = p;
        s_prim[group][c] = x.prims[p];
      }
      __syncwarp(gmask);
      const uint32_t m = min(8u, it.pcount - k0);
      for (uint32_t j = 0; j < m; ++j) {
        const uint32_t k = k0 + j;
        const uint32_t cls =
            pol.template classify<Terrain>(s_prim[group][j], world_exp, ox, oy, oz, csize);
        if (cls == VX_CELL_FULL) {
          last_full = static_cast<int32_t>(s_pidx[group][j]);
          cnt = 0;
          partial = 0;
        } else if (cls == VX_CELL_MIXED) {
          left.add(s_prim[group][j], cnt == 0);
          ++cnt;
          if (k < 32u) partial |= 1u << k;
        }
      }
      __syncwarp(gmask); // the chunk is overwritten next
    }
    const uint32_t const_val =
        last_full >= 0 ? pol.const_value(x.prims[last_full], oz, csize) : 0u;
    if (!Terrain && cnt != 0 && left.all(pol, last_full >= 0 ? const_val : old_child)) cnt = 0;
    // Prefix sums over the 8 lanes of the group.
    uint32_t inc_items =
                 (cnt != 0 || (Policy::kItemsForConst && last_full >= 0)) ? 1u : 0u,
             inc_pairs = cnt;
#pragma unroll
    for (uint32_t d = 1; d < 8; d <<= 1) {
      const uint32_t a = __shfl_up_sync(kFullMask, inc_items, d, 8);
      const uint32_t b = __shfl_up_sync(kFullMask, inc_pairs, d, 8);
      if (c >= d) {
        inc_items += a;
        inc_pairs += b;
      }
    }
    const uint32_t group_items = __shfl_sync(kFullMask, inc_items, 7, 8);
    const uint32_t group_pairs = __shfl_sync(kFullMask, inc_pairs, 7, 8);
    const bool full_add = last_full >= 0 && const_val == 1u;
    const bool has_item = cnt != 0 || (Policy::kItemsForConst && last_full >= 0);
    const uint32_t child_mask = (__ballot_sync(kFullMask, has_item) >> gshift) & 0xffu;
    const uint32_t const_mask = (__ballot_sync(kFullMask, last_full >= 0) >> gshift) & 0xffu;
    const uint32_t const_full = (__ballot_sync(kFullMask, full_add) >> gshift) & 0xffu;
    if (c == 0) {
      s_items[group] = have && !big ? group_items : 0u;
      s_pairs[group] = have && !big ? group_pairs : 0u;
    }
    __syncthreads();
    if (threadIdx.x < kWarp) { // one group per lane: exclusive offsets by shuffles
      const uint32_t a = s_items[threadIdx.x], b = s_pairs[threadIdx.x];
      const uint32_t ia = warp_inclusive_sum(a), ib = warp_inclusive_sum(b);
      s_items[threadIdx.x] = ia - a;
      s_pairs[threadIdx.x] = ib - b;
      const uint32_t ti = __shfl_sync(kFullMask, ia, kWarp - 1);
      const uint32_t tp = __shfl_sync(kFullMask, ib, kWarp - 1);
      if (threadIdx.x == 0) {
        s_item_base = ti ? atomicAdd(&h->item_count[l + 1], ti) : 0;
        s_pair_base = tp ? atomicAdd(&h->pair_count[l + 1], tp) : 0;
        // this tile's own room (an overflow elsewhere fails the edit at the
        // next stage; writing within the buffers meanwhile is harmless)
        bool room = true;
        if (ti && static_cast<uint64_t>(next_base) + s_item_base + ti > x.a.item_cap) room = false;
        if (tp && static_cast<uint64_t>(s_pair_base) + tp > x.a.pair_cap) room = false;
        if (!room) set_status(&h->status, kDevCapacity);
        s_room = room;
      }
    }
    __syncthreads();
    const bool room = s_room;
    const uint32_t item_off = s_item_base + s_items[group];
    const uint32_t pair_off = s_pair_base + s_pairs[group];
    __syncthreads(); // s_* are reused by the next tile
    if (!have || big || !room) continue;
    if (last_full >= 0) pol.replaced(l, it.old, c);

    if (has_item) {
      const uint32_t my_pairs = pair_off + inc_pairs - cnt;
      Item ci{};
      ci.cell = child_cell(it.cell, c);
      ci.old = last_full >= 0 ? const_val : old_child;
      ci.pstart = my_pairs;
      ci.pcount = cnt;
      ci.result = static_cast<uint32_t>(base + wi);
      x.a.items[next_base + item_off + inc_items - 1] = ci;
      note_big(x, l + 1, item_off + inc_items - 1, cnt);
      uint32_t j = 0;
      if (it.pcount <= 32u) {
        // The child's list is the set bits of `partial`: independent loads
        // of the pairs, no second classification.
        for (uint32_t bits = cnt ? partial : 0u; bits != 0u; bits &= bits - 1u)
          out_pairs[my_pairs + j++] = in_pairs[it.pstart + __ffs(bits) - 1u];
      } else {
        for (uint32_t k = 0; k < it.pcount && j < cnt; ++k) {
          const uint32_t p = in_pairs[it.pstart + k];
          if (static_cast<int32_t>(p) <= last_full) continue;
          if (pol.template classify<Terrain>(x.prims[p], world_exp, ox, oy, oz, csize) == VX_CELL_MIXED)
            out_pairs[my_pairs + j++] = p;
        }
      }
    }
    if (c == 0) {
      x.a.items[base + wi].child_base = next_base + item_off;
      x.a.items[base + wi].masks = child_mask | (const_mask << 8) | (const_full << 16);
      x.a.items[base + wi].pstart = __popc(child_mask); // the pairs were read above
    }
  }
}

template <class Policy, bool Terrain>
__global__ void __launch_bounds__(kBlock)
    expand_kernel(EditCtx x, Policy pol, uint32_t l) {
  expand_body<Policy, Terrain>(x, pol, l, launch_blocks());
}

// Up to this many items a level's batch kernels (expand, leaf parents) give
// eight lanes to an item instead of one: so many are on the chip at once, and
// a warp that takes 32 items with several primitives each would walk their
// lists four (expansion) or a leaf at a time (leaf parents) while most of the
// chip has nothing to do.  B200, us, one lane / eight lanes up to here (eight
// always): 2,000 spheres of radius 16-64 with their centres in a 256^3 part
// of a 2048^3 Hash DAG 620 / 369 (453), of an SVO 578 / 371 (594); 1,000
// primitives in a 256^3 world 393 / 187 (287); 8,000 spheres all over 2048^3
// 592 / 463 (893).
constexpr uint32_t kWideItems = 37888; // 148 multiprocessors x 256 groups of eight

// expand_body for the batches' own launches: a warp takes 32 items at a time
// with no block barrier.  At the levels that hold most items nearly every
// list is one primitive (at 16,384 spheres in 16384^3, 6.67 M primitives for
// 6.65 M items two levels above the leaves), so each lane owns an item: its
// record, its primitive, all eight children's classification and previous
// contents.  Items with more primitives (up to big_item) then get eight
// lanes each, four at a time, as in expand_body.  The warp takes room for all
// its children with one atomic per counter, and the children are listed and
// dealt out to the lanes, so that 32 child items go out as one contiguous
// write.
// On B200: 1.82 -> 0.89 ms for the levels of that batch (9.0 M items).
struct ExpandWarp {
  uint32_t ref[8][kWarp];     // [child][item]: what the child starts from
  uint32_t list[8][kWarp];    // several primitives: which of the first 32 go down, or
                              // (longer lists) 1 + the last covering primitive
  uint32_t span[8][kWarp];    // several: how many go down | offset in the item's pairs << 16
  uint32_t verdict[kWarp];    // several: child items | covered << 8 | covered and full << 16
  uint32_t npairs[kWarp];     // several: pairs of all children
  uint32_t pidx[4][8];        // the four groups' current chunks of their lists
  vx_primitive prim[4][8];
  uint8_t task[8 * kWarp];    // item | child << 5
};

template <class Policy>
__global__ void __launch_bounds__(kBlock, 4) expand_warp_kernel(EditCtx x, Policy pol, uint32_t l) {
  __shared__ ExpandWarp s_warp[kBlock / kWarp];
  Header *h = x.hdr;
  const uint32_t W = h->item_count[l]; // loaded beside the status
  const uint32_t base = h->item_off[l];
  if (W <= kWideItems) { // the same in every block
    expand_body<Policy, false>(x, pol, l, launch_blocks());
    return;
  }
  if (edit_failed(h)) return;
  const uint32_t depth = x.depth;
  const uint32_t next_base = base + W;
  if (blockIdx.x == 0 && threadIdx.x == 0) h->item_off[l + 1] = next_base;
  const uint32_t *in_pairs = x.a.pairs[l & 1u];
  uint32_t *out_pairs = x.a.pairs[(l + 1) & 1u];
  const uint32_t csize = 4u << (depth - l - 1); // child cell side
  const uint32_t world_exp = depth + 2;
  const uint32_t lane = lane_id();
  const uint32_t group = lane >> 3, gc = lane & 7u; // for items with several primitives
  const uint32_t gshift = lane & ~7u;
  const uint32_t gmask = 0xffu << gshift;
  ExpandWarp &s = s_warp[threadIdx.x / kWarp];

  for (uint64_t w0 = blockIdx.x * uint64_t(kBlock) + threadIdx.x - lane; w0 < W;
       w0 += uint64_t(gridDim.x) * kBlock) {
    const uint32_t wi = static_cast<uint32_t>(w0) + lane;
    const bool have = w0 + lane < W;
    Item it{};
    if (have) it = x.a.items[base + wi];
    // Items with long lists were listed when they were emitted (big_list).
    const bool big = have && it.pcount > x.big_item;
    const bool single = have && it.pcount == 1u;
    uint32_t v = 0, npairs = 0, pidx = 0;
    if (single) {
      pidx = in_pairs[it.pstart];
      uint32_t ref[8];
      pol.children(l, it.old, ref);
      const vx_primitive pr = x.prims[pidx];
      uint32_t touched, covered;
      if (vx_prim_shape(&pr) == VX_SHAPE_SPHERE && pr.r[0] < kFastRadius) {
        const Cell cell = unpack_cell(it.cell);
        sphere_classify_children(pr, cell.x * 2u * csize, cell.y * 2u * csize, cell.z * 2u * csize,
                                 csize, touched, covered);
      } else {
        const uint32_t tc = other_children(x.prims + pidx, it.cell, csize);
        touched = tc & 0xffu;
        covered = tc >> 8;
      }
      const uint32_t cv = pol.const_value(pr, 0, csize);
      uint32_t held = 0; // children that hold just that everywhere (LeftValue)
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        s.ref[c][lane] = (covered >> c) & 1u ? cv : ref[c];
        if (ref[c] == cv) held |= 1u << c;
      }
      for (uint32_t m = covered; m != 0u; m &= m - 1u) pol.replaced(l, it.old, __ffs(m) - 1u);
      const uint32_t mixed = touched & ~covered & ~held;
      v = mixed | (Policy::kItemsForConst ? covered : 0u) | (covered << 8) |
          (cv == 1u ? covered << 16 : 0u);
      npairs = __popc(mixed);
    }
    // Items with several primitives, four at a time: lane gc of a group takes
    // child gc, the group stages its list eight primitives at a time.
    const bool several = have && !big && it.pcount > 1u;
    const uint32_t all_several = __ballot_sync(kFullMask, several);
    for (uint32_t left = all_several; left != 0u;) {
      uint32_t mine = left;
      for (uint32_t g = 0; g < group; ++g) mine &= mine - 1u;
      for (uint32_t g = 0; g < 4u; ++g) left &= left - 1u; // (0 stays 0)
      const bool on = mine != 0u;
      const uint32_t src = on ? __ffs(mine) - 1u : 0u;
      const uint64_t cell_bits = __shfl_sync(kFullMask, it.cell, src);
      const uint32_t old = __shfl_sync(kFullMask, it.old, src);
      const uint32_t pstart = __shfl_sync(kFullMask, it.pstart, src);
      const uint32_t count = __shfl_sync(kFullMask, it.pcount, src);
      const uint32_t pcount = on ? count : 0u;
      const Cell cell = unpack_cell(cell_bits);
      const int64_t ox = int64_t(2 * cell.x + (gc & 1u)) * csize;
      const int64_t oy = int64_t(2 * cell.y + ((gc >> 1) & 1u)) * csize;
      const int64_t oz = int64_t(2 * cell.z + (gc >> 2)) * csize;
      const uint32_t old_child = on ? pol.child(l, old, gc) : 0u;
      int32_t last_full = -1;
      uint32_t cnt = 0, partial = 0; // as in expand_body
      LeftValue<Policy> kept;
      for (uint32_t k0 = 0; k0 < pcount; k0 += 8) {
        if (k0 + gc < pcount) {
          const uint32_t p = in_pairs[pstart + k0 + gc];
          s.pidx[group][gc] = p;
          s.prim[group][gc] = x.prims[p];
        }
        __syncwarp(gmask);
        const uint32_t m = min(8u, pcount - k0);
        for (uint32_t j = 0; j < m; ++j) {
          const uint32_t k = k0 + j;
          const uint32_t cls =
              pol.template classify<false>(s.prim[group][j], world_exp, ox, oy, oz, csize);
          if (cls == VX_CELL_FULL) {
            last_full = static_cast<int32_t>(s.pidx[group][j]);
            cnt = 0;
            partial = 0;
          } else if (cls == VX_CELL_MIXED) {
            kept.add(s.prim[group][j], cnt == 0);
            ++cnt;
            if (k < 32u) partial |= 1u << k;
          }
        }
        __syncwarp(gmask); // the chunk is overwritten next
      }
      __syncwarp();
      const bool covered = last_full >= 0;
      const uint32_t cv = covered ? pol.const_value(x.prims[last_full], oz, csize) : 0u;
      if (covered) pol.replaced(l, old, gc);
      if (cnt != 0 && kept.all(pol, covered ? cv : old_child)) cnt = partial = 0;
      uint32_t inc = cnt;
#pragma unroll
      for (uint32_t d = 1; d < 8; d <<= 1) {
        const uint32_t o = __shfl_up_sync(kFullMask, inc, d, 8);
        if (gc >= d) inc += o;
      }
      const uint32_t child_mask =
          __ballot_sync(kFullMask, cnt != 0 || (Policy::kItemsForConst && covered)) >> gshift;
      const uint32_t const_mask = __ballot_sync(kFullMask, covered) >> gshift;
      const uint32_t full_mask = __ballot_sync(kFullMask, covered && cv == 1u) >> gshift;
      if (on) {
        s.ref[gc][src] = covered ? cv : old_child;
        s.list[gc][src] = pcount <= 32u ? partial : static_cast<uint32_t>(last_full + 1);
        s.span[gc][src] = cnt | ((inc - cnt) << 16);
        if (gc == 7u) s.npairs[src] = inc;
        if (gc == 0u)
          s.verdict[src] =
              (child_mask & 0xffu) | ((const_mask & 0xffu) << 8) | ((full_mask & 0xffu) << 16);
      }
    }
    __syncwarp();
    if (several) {
      v = s.verdict[lane];
      npairs = s.npairs[lane];
    }
    // Room for the warp's children and their pairs.
    const uint32_t nitems = __popc(v & 0xffu);
    const uint32_t inc_items = warp_inclusive_sum(nitems), inc_pairs = warp_inclusive_sum(npairs);
    uint32_t item_at = 0, pair_at = 0;
    bool room = true;
    if (lane == kWarp - 1) {
      if (inc_items) item_at = atomicAdd(&h->item_count[l + 1], inc_items);
      if (inc_pairs) pair_at = atomicAdd(&h->pair_count[l + 1], inc_pairs);
      // this warp's own room (an overflow elsewhere fails the edit at the
      // next stage; writing within the buffers meanwhile is harmless)
      room = !(inc_items && uint64_t(next_base) + item_at + inc_items > x.a.item_cap) &&
             !(inc_pairs && uint64_t(pair_at) + inc_pairs > x.a.pair_cap);
      if (!room) set_status(&h->status, kDevCapacity);
    }
    const uint32_t tasks = __shfl_sync(kFullMask, inc_items, kWarp - 1);
    item_at = __shfl_sync(kFullMask, item_at, kWarp - 1);
    pair_at = __shfl_sync(kFullMask, pair_at, kWarp - 1) + inc_pairs - npairs;
    if (!__shfl_sync(kFullMask, room ? 1 : 0, kWarp - 1)) continue;
    const uint32_t my_item = item_at + inc_items - nitems; // first child, within its level
    if (have && !big) {
      Item &me = x.a.items[base + wi];
      me.child_base = next_base + my_item;
      me.masks = v;
      me.pstart = nitems; // the pairs were read above, or are held by `it`
    }
    uint32_t at = inc_items - nitems;
    for (uint32_t m = v & 0xffu; m != 0u; m &= m - 1u)
      s.task[at++] = static_cast<uint8_t>(lane | ((__ffs(m) - 1u) << 5));
    __syncwarp();
    for (uint32_t t0 = 0; t0 < tasks; t0 += kWarp) {
      const bool busy = t0 + lane < tasks;
      const uint32_t task = busy ? s.task[t0 + lane] : 0u;
      const uint32_t src = task & 31u, c = task >> 5;
      const uint64_t cell_bits = __shfl_sync(kFullMask, it.cell, src);
      const uint32_t sv = __shfl_sync(kFullMask, v, src);
      const uint32_t pairs0 = __shfl_sync(kFullMask, pair_at, src);
      const uint32_t prim = __shfl_sync(kFullMask, pidx, src);
      if (!busy) continue;
      const bool one = ((all_several >> src) & 1u) == 0u;
      Item ci{};
      ci.cell = child_cell(cell_bits, c);
      ci.old = s.ref[c][src];
      if (one) { // its one primitive cuts every child that it does not cover
        const uint32_t mixed = sv & ~(sv >> 8) & 0xffu;
        ci.pcount = (mixed >> c) & 1u;
        ci.pstart = pairs0 + __popc(mixed & ((1u << c) - 1u));
        if (ci.pcount) out_pairs[ci.pstart] = prim;
      } else {
        const uint32_t span = s.span[c][src];
        ci.pcount = span & 0xffffu;
        ci.pstart = pairs0 + (span >> 16);
        note_big(x, l + 1, item_at + t0 + lane, ci.pcount);
      }
      ci.result = base + static_cast<uint32_t>(w0) + src;
      x.a.items[next_base + item_at + t0 + lane] = ci;
    }
    // The lists of the children of items with several primitives.
    for (uint32_t left = all_several; left != 0u;) {
      uint32_t mine = left;
      for (uint32_t g = 0; g < group; ++g) mine &= mine - 1u;
      for (uint32_t g = 0; g < 4u; ++g) left &= left - 1u;
      const bool on = mine != 0u;
      const uint32_t src = on ? __ffs(mine) - 1u : 0u;
      const uint64_t cell_bits = __shfl_sync(kFullMask, it.cell, src);
      const uint32_t pstart = __shfl_sync(kFullMask, it.pstart, src);
      const uint32_t pcount = __shfl_sync(kFullMask, it.pcount, src);
      const uint32_t pairs0 = __shfl_sync(kFullMask, pair_at, src);
      if (!on) continue;
      const uint32_t span = s.span[gc][src];
      const uint32_t cnt = span & 0xffffu;
      uint32_t to = pairs0 + (span >> 16);
      if (pcount <= 32u) {
        for (uint32_t bits = s.list[gc][src]; bits != 0u; bits &= bits - 1u)
          out_pairs[to++] = in_pairs[pstart + __ffs(bits) - 1u];
        continue;
      }
      const int32_t last_full = static_cast<int32_t>(s.list[gc][src]) - 1;
      const Cell cell = unpack_cell(cell_bits);
      const int64_t ox = int64_t(2 * cell.x + (gc & 1u)) * csize;
      const int64_t oy = int64_t(2 * cell.y + ((gc >> 1) & 1u)) * csize;
      const int64_t oz = int64_t(2 * cell.z + (gc >> 2)) * csize;
      const uint32_t end = to + cnt;
      for (uint32_t k = 0; k < pcount && to < end; ++k) {
        const uint32_t p = in_pairs[pstart + k];
        if (static_cast<int32_t>(p) <= last_full) continue;
        if (pol.template classify<false>(x.prims[p], world_exp, ox, oy, oz, csize) ==
            VX_CELL_MIXED)
          out_pairs[to++] = p;
      }
    }
    __syncwarp(); // the next items overwrite the warp's buffers
  }
}

// Expansion of level l for primitives that are the leaf masks of distinct
// leaves in leaf key order (a sorted voxel list or sorted leaf commands): the
// primitives inside a cell are a contiguous range of the list, so an item
// needs no list walk and no pair lists, only the borders between its
// children.  Eight lanes per item, lane c searching the first primitive at or
// after child c's key range; the pair buffers hold the identity (init_body),
// so later stages read the lists as usual.  A leaf mask never covers a cell
// above the leaves, so no child is constant.
//
// Walking the lists costs time in proportion to the list at every level whose
// cells hold most of it, on one block per cell: the 144,000 leaves of a
// sphere of radius 128 in a 4096^3 world took a block per cell 5.8 ms (and
// the short lists 0.18 ms) of an edit's 7.0 ms on B200, the searches 0.10 ms (by
// halves 0.13): a chain of log8(list) round trips to L2 per level.
template <class Policy>
__device__ __forceinline__ void expand_sorted_body(EditCtx x, Policy pol, uint32_t l, Blocks blk) {
  Header *h = x.hdr;
  const uint32_t W = h->item_count[l];
  const uint32_t base = h->item_off[l];
  if (edit_failed(h)) return;
  const uint32_t next_base = base + W;
  if (blk.id == 0 && threadIdx.x == 0) {
    h->item_off[l + 1] = next_base;
    h->pair_count[l + 1] = h->pair_count[l]; // a leaf goes on to one child at most
  }
  const uint64_t *keys = x.sorted_keys;
  const uint32_t item_shift = 3 * (x.depth - l);
  const uint32_t lane = lane_id(), c = lane & 7u;
  const uint32_t gshift = lane & ~7u;
  const uint64_t total = static_cast<uint64_t>(W) * 8u;
  const uint64_t stride = static_cast<uint64_t>(blk.count) * blockDim.x;
  for (uint64_t g0 = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x - lane; g0 < total;
       g0 += stride) {
    const uint32_t wi = static_cast<uint32_t>((g0 + lane) >> 3);
    const bool have = wi < W;
    Item it{};
    uint32_t lo = 0, old_child = 0;
    if (have) {
      it = x.a.items[base + wi];
      old_child = pol.child(l, it.old, c);
      // first primitive whose key is at or after child c's first leaf
      const uint64_t want = ((keys[it.pstart] >> item_shift) << item_shift) |
                            (static_cast<uint64_t>(c) << (item_shift - 3u));
      // Seven probes a round, loaded together: a third of a binary search's
      // chain of round trips on the long lists of the top levels.
      lo = it.pstart;
      uint32_t n = it.pcount;
      while (n != 0) {
        const uint32_t step = n / 8u + 1u; // probes at lo + step - 1, lo + 2 step - 1, ...
        uint64_t k[7];
#pragma unroll
        for (uint32_t j = 0; j < 7; ++j)
          k[j] = (j + 1) * step <= n ? keys[lo + (j + 1) * step - 1] : ~0ull;
        uint32_t below = 0; // probes below `want` (they ascend)
#pragma unroll
        for (uint32_t j = 0; j < 7; ++j) below += k[j] < want ? 1u : 0u;
        lo += below * step;
        n = min(n - below * step, step - 1u);
      }
    }
    const uint32_t next = __shfl_down_sync(kFullMask, lo, 1, 8);
    uint32_t cnt = have ? (c == 7u ? it.pstart + it.pcount : next) - lo : 0u;
    // One operation for the whole list: a child that holds its value everywhere
    // stays as it is (LeftValue).
    if (cnt != 0 && old_child == pol.const_value(x.prims[lo], 0, 4)) cnt = 0;
    const uint32_t some = __ballot_sync(kFullMask, cnt != 0);
    const uint32_t child_mask = (some >> gshift) & 0xffu;
    uint32_t first = 0; // one atomic per warp: four items' children
    if (lane == 0 && some) first = atomicAdd(&h->item_count[l + 1], __popc(some));
    first = __shfl_sync(kFullMask, first, 0);
    if (static_cast<uint64_t>(next_base) + first + __popc(some) > x.a.item_cap) {
      if (lane == 0) set_status(&h->status, kDevCapacity);
      continue;
    }
    if (cnt != 0) {
      Item ci{};
      ci.cell = child_cell(it.cell, c);
      ci.old = old_child;
      ci.pstart = lo;
      ci.pcount = cnt;
      ci.result = base + wi;
      x.a.items[next_base + first + __popc(some & lanemask_lt())] = ci;
    }
    if (have && c == 0) {
      Item &me = x.a.items[base + wi];
      me.child_base = next_base + first + __popc(some & lanemask_lt());
      me.masks = child_mask;
      me.pstart = __popc(child_mask);
    }
  }
}

template <class Policy>
__global__ void __launch_bounds__(kBlock) expand_sorted_kernel(EditCtx x, Policy pol, uint32_t l) {
  expand_sorted_body<Policy>(x, pol, l, launch_blocks());
}

// Blocks for a stage over level l's items with `per_block` items a block:
// level l holds at most 8^l of them, and a launch of thousands of blocks that
// find nothing to do takes 6 us, one of a few blocks 2.
inline uint32_t level_grid(uint32_t grid, uint32_t l, uint32_t per_block) {
  if (l >= 10) return grid;
  const uint32_t need = ceil_div(uint64_t(1) << (3 * l), per_block);
  return need < grid ? need : grid;
}

// Blocks of expand_warp_kernel for level l: 256 items a block, or 32 while the
// level has so few that it takes the eight-lane body.
inline uint32_t expand_grid(uint32_t grid, uint32_t l) {
  return std::max(level_grid(grid, l, kBlock),
                  std::min(level_grid(grid, l, kBlock / 8), ceil_div(kWideItems, kBlock / 8)));
}

// Expansion of the long-list items of level l inside the small cooperative
// kernels: one block of Threads threads per item.  Three walks over the list:
// the last fully-covering primitive per child (block max), the partial
// primitives after it per child (block sum), then an order-preserving
// block-wide compaction of those into each child's list.  Lists of up to
// Cache primitives are classified once: walk 1 keeps each primitive's
// per-child MIXED bits in shared memory for walks 2 and 3.
template <class Policy, uint32_t Threads, uint32_t Cache>
__device__ __forceinline__ void expand_big_body(EditCtx x, Policy pol, uint32_t l, Blocks blk) {
  Header *h = x.hdr;
  // the level's counts and this block's first listed item load beside the
  // status (the list is read past its count only within its buffer)
  const uint32_t nbig = min(h->big_count[l], x.a.big_cap / 2u);
  const uint32_t *bigs = big_list(x.a, l);
  const uint32_t base = h->item_off[l];
  const uint32_t next_base = base + h->item_count[l];
  uint32_t first_wi = blk.id < x.a.big_cap / 2u ? bigs[blk.id] : 0u;
  if (edit_failed(h)) return;
  const uint32_t depth = x.depth;
  const uint32_t *in_pairs = x.a.pairs[l & 1u];
  uint32_t *out_pairs = x.a.pairs[(l + 1) & 1u];
  const int64_t csize = int64_t(4) << (depth - l - 1);
  const uint32_t world_exp = depth + 2;
  constexpr uint32_t kWarps = Threads / kWarp;
  static_assert(kWarps <= kWarp, "one warp scans the warps' counts");
  __shared__ int32_t s_last[8];
  __shared__ uint32_t s_cnt[8], s_start[8], s_const[8], s_cm;
  __shared__ uint32_t s_warp[8][kWarps], s_total[8];
  __shared__ uint32_t s_item_base, s_pair_base;
  __shared__ bool s_room;
  __shared__ uint8_t s_mixed[Cache];
  const uint32_t t = threadIdx.x, lane = lane_id(), warp = t / kWarp;

  for (uint32_t b = blk.id; b < nbig; b += blk.count) {
    const uint32_t wi = b == blk.id ? first_wi : bigs[b];
    const Item it = x.a.items[base + wi];
    const Cell cell = unpack_cell(it.cell);
    const bool cached = it.pcount <= Cache; // block-uniform
    // child t's previous content, loaded beside the walks (used unless a
    // primitive covers the child)
    const uint32_t old_child = t < 8 ? pol.child(l, it.old, t) : 0u;
    if (t < 8) {
      s_last[t] = -1;
      s_cnt[t] = 0;
    }
    __syncthreads();
    // Walk 1: last FULL per child (and the MIXED bits, when cached).
    int32_t last[8];
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) last[c] = -1;
    for (uint32_t k = t; k < it.pcount; k += Threads) {
      const uint32_t p = in_pairs[it.pstart + k];
      const vx_primitive pr = x.prims[p];
      uint32_t mixed = 0;
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        const int64_t ox = int64_t(2 * cell.x + (c & 1u)) * csize;
        const int64_t oy = int64_t(2 * cell.y + ((c >> 1) & 1u)) * csize;
        const int64_t oz = int64_t(2 * cell.z + ((c >> 2) & 1u)) * csize;
        const uint32_t cls = pol.template classify<false>(pr, world_exp, ox, oy, oz, csize);
        if (cls == VX_CELL_FULL) last[c] = max(last[c], static_cast<int32_t>(p));
        else if (cls == VX_CELL_MIXED) mixed |= 1u << c;
      }
      if (cached) s_mixed[k] = static_cast<uint8_t>(mixed);
    }
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      const int32_t m = __reduce_max_sync(kFullMask, last[c]);
      if (lane == 0 && m >= 0) atomicMax(&s_last[c], m);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) last[c] = s_last[c];
    // Walk 2: partial primitives after the last full one.
    uint32_t cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t k = t; k < it.pcount; k += Threads) {
      const uint32_t p = in_pairs[it.pstart + k];
      if (cached) { // each thread reads back the bits it wrote in walk 1
        const uint32_t mixed = s_mixed[k];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c)
          cnt[c] += (static_cast<int32_t>(p) > last[c] && ((mixed >> c) & 1u)) ? 1u : 0u;
        continue;
      }
      const vx_primitive pr = x.prims[p];
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        if (static_cast<int32_t>(p) <= last[c]) continue;
        const int64_t ox = int64_t(2 * cell.x + (c & 1u)) * csize;
        const int64_t oy = int64_t(2 * cell.y + ((c >> 1) & 1u)) * csize;
        const int64_t oz = int64_t(2 * cell.z + ((c >> 2) & 1u)) * csize;
        if (pol.template classify<false>(pr, world_exp, ox, oy, oz, csize) == VX_CELL_MIXED) ++cnt[c];
      }
    }
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      const uint32_t v = __reduce_add_sync(kFullMask, cnt[c]);
      if (lane == 0 && v) atomicAdd(&s_cnt[c], v);
    }
    __syncthreads();
    if (t == 0) {
      uint32_t ni = 0, np = 0, cm = 0, km = 0, kf = 0;
      for (uint32_t c = 0; c < 8; ++c) {
        s_start[c] = np;
        const int64_t coz = int64_t(2 * cell.z + ((c >> 2) & 1u)) * csize;
        s_const[c] = s_last[c] >= 0 ? pol.const_value(x.prims[s_last[c]], coz, csize) : 0u;
        if (s_cnt[c] || (Policy::kItemsForConst && s_last[c] >= 0)) {
          cm |= 1u << c;
          ++ni;
          np += s_cnt[c];
        }
        if (s_last[c] >= 0) {
          km |= 1u << c;
          if (s_const[c] == 1u) kf |= 1u << c;
        }
      }
      s_cm = cm;
      s_item_base = ni ? atomicAdd(&h->item_count[l + 1], ni) : 0;
      s_pair_base = np ? atomicAdd(&h->pair_count[l + 1], np) : 0;
      // this item's own room (an overflow elsewhere fails the edit at the
      // next stage; writing within the buffers meanwhile is harmless)
      bool room = true;
      if (ni && static_cast<uint64_t>(next_base) + s_item_base + ni > x.a.item_cap) room = false;
      if (np && static_cast<uint64_t>(s_pair_base) + np > x.a.pair_cap) room = false;
      if (!room) set_status(&h->status, kDevCapacity);
      x.a.items[base + wi].child_base = next_base + s_item_base;
      x.a.items[base + wi].masks = cm | (km << 8) | (kf << 16);
      x.a.items[base + wi].pstart = __popc(cm); // every thread holds its own copy of it
      s_room = room;
    }
    __syncthreads();
    const bool room = s_room; // block-uniform: it guards barriers below
    if (room && t < 8 && s_last[t] >= 0) pol.replaced(l, it.old, t);
    if (room && t < 8 && ((s_cm >> t) & 1u)) {
      const uint32_t k = __popc(s_cm & ((1u << t) - 1u));
      Item ci{};
      ci.cell = child_cell(it.cell, t);
      ci.old = s_last[t] >= 0 ? s_const[t] : old_child;
      ci.pstart = s_pair_base + s_start[t];
      ci.pcount = s_cnt[t];
      ci.result = static_cast<uint32_t>(base + wi);
      x.a.items[next_base + s_item_base + k] = ci;
      note_big(x, l + 1, s_item_base + k, s_cnt[t]);
    }
    // Walk 3: order-preserving compaction, one Threads-pair chunk at a time.
    uint32_t run[8];
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) run[c] = s_pair_base + s_start[c];
    for (uint32_t k0 = 0; k0 < it.pcount && room; k0 += Threads) {
      const uint32_t k = k0 + t;
      uint32_t take = 0, p = 0;
      if (k < it.pcount && cached) {
        p = in_pairs[it.pstart + k];
        const uint32_t mixed = s_mixed[k];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c)
          if (static_cast<int32_t>(p) > last[c] && ((mixed >> c) & 1u)) take |= 1u << c;
      } else if (k < it.pcount) {
        p = in_pairs[it.pstart + k];
        const vx_primitive pr = x.prims[p];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) {
          if (static_cast<int32_t>(p) <= last[c]) continue;
          const int64_t ox = int64_t(2 * cell.x + (c & 1u)) * csize;
          const int64_t oy = int64_t(2 * cell.y + ((c >> 1) & 1u)) * csize;
          const int64_t oz = int64_t(2 * cell.z + ((c >> 2) & 1u)) * csize;
          if (pol.template classify<false>(pr, world_exp, ox, oy, oz, csize) == VX_CELL_MIXED)
            take |= 1u << c;
        }
      }
      uint32_t ballots[8];
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        ballots[c] = __ballot_sync(kFullMask, (take >> c) & 1u);
        if (lane == 0) s_warp[c][warp] = __popc(ballots[c]);
      }
      __syncthreads();
      if (warp == 0) { // exclusive offsets of the warps, per child, by shuffles
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) {
          const uint32_t v = lane < kWarps ? s_warp[c][lane] : 0u;
          const uint32_t inc = warp_inclusive_sum(v);
          if (lane < kWarps) s_warp[c][lane] = inc - v;
          if (lane == kWarp - 1) s_total[c] = inc;
        }
      }
      __syncthreads();
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        if ((take >> c) & 1u)
          out_pairs[run[c] + s_warp[c][warp] + __popc(ballots[c] & lanemask_lt())] = p;
        run[c] += s_total[c];
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

// The same for the batches' own launches.  A list longer than kLongList is
// expanded by a cluster of eight blocks (the root of a batch carries every
// primitive), a shorter one by one block.  Each warp owns a contiguous part
// of the list, so its order is kept without a barrier per step: the three
// walks are separated by one exchange each (the covering primitive per child,
// the counts per warp and child, the room taken), over the blocks' shared
// memory inside a cluster.  Classification treats a primitive's eight children
// together and is kept as a byte per primitive for the later walks.
// On B200, nine levels of two batches of 32,768 primitives: 1.18 -> 0.48 ms;
// eleven levels of 16,384 spheres: 0.27 -> 0.14 ms.
constexpr uint32_t kLongBlock = 512, kLongCluster = 8, kLongList = 4096;
constexpr uint32_t kLongWarps = kLongBlock / kWarp;
constexpr uint32_t kLongCache = 32768; // primitives per block whose bits are kept

struct LongShared {
  uint8_t mixed[kLongCache];
  int32_t warp_last[kLongWarps][8];
  uint32_t warp_count[kLongWarps][8]; // then each warp's offset in its block
  int32_t last[kLongCluster][8];      // per block of the cluster
  uint32_t count[kLongCluster][8];
  uint32_t at[8];                     // first pair of each child's list
  uint32_t room;
  uint32_t failed[kLongCluster];
};

template <class Policy, uint32_t Cl>
__device__ __forceinline__ void expand_long_item(const EditCtx &x, const Policy &pol, uint32_t l,
                                                 uint32_t wi, uint32_t base, uint32_t next_base,
                                                 LongShared &s) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = Cl > 1 ? cluster.block_rank() : 0u;
  auto sync_all = [&]() {
    if constexpr (Cl > 1) cluster.sync();
    else __syncthreads();
  };
  // v into *field of every block of the cluster
  auto share = [&](auto *field, auto v) {
    if constexpr (Cl > 1) {
      for (uint32_t r = 0; r < Cl; ++r) *cluster.map_shared_rank(field, r) = v;
    } else {
      *field = v;
    }
  };
  Header *h = x.hdr;
  const uint32_t t = threadIdx.x, lane = lane_id(), warp = t / kWarp;
  const uint32_t *in_pairs = x.a.pairs[l & 1u];
  uint32_t *out_pairs = x.a.pairs[(l + 1) & 1u];
  const uint32_t csize = 4u << (x.depth - l - 1);
  const Item it = x.a.items[base + wi];
  const uint32_t units = (it.pcount + kWarp - 1) / kWarp;
  const uint32_t part = (units + Cl * kLongWarps - 1) / (Cl * kLongWarps) * kWarp; // per warp
  const uint32_t block_first = rank * kLongWarps * part;
  const uint32_t first = min(block_first + warp * part, it.pcount);
  const uint32_t end = min(first + part, it.pcount);
  const bool cached = kLongWarps * part <= kLongCache;
  const uint32_t old_child = rank == 0 && t < 8 ? pol.child(l, it.old, t) : 0u;
  const Cell cell = unpack_cell(it.cell);
  auto classify8 = [&](uint32_t p, uint32_t &touched, uint32_t &covered) {
    const vx_primitive pr = x.prims[p];
    if (vx_prim_shape(&pr) == VX_SHAPE_SPHERE && pr.r[0] < kFastRadius) {
      sphere_classify_children(pr, cell.x * 2u * csize, cell.y * 2u * csize, cell.z * 2u * csize,
                               csize, touched, covered);
    } else {
      const uint32_t tc = other_children(x.prims + p, it.cell, csize);
      touched = tc & 0xffu;
      covered = tc >> 8;
    }
  };
  // Walk 1: the last covering primitive per child.
  int32_t last[8];
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) last[c] = -1;
  for (uint32_t k = first + lane; k < end; k += kWarp) {
    const uint32_t p = in_pairs[it.pstart + k];
    uint32_t touched, covered;
    classify8(p, touched, covered);
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      if ((covered >> c) & 1u) last[c] = static_cast<int32_t>(p); // lists ascend
    if (cached) s.mixed[k - block_first] = static_cast<uint8_t>(touched & ~covered);
  }
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    const int32_t m = __reduce_max_sync(kFullMask, last[c]);
    if (lane == 0) s.warp_last[warp][c] = m;
  }
  __syncthreads();
  if (t < 8) {
    int32_t m = -1;
    for (uint32_t w = 0; w < kLongWarps; ++w) m = max(m, s.warp_last[w][t]);
    share(&s.last[rank][t], m);
  }
  sync_all();
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    last[c] = s.last[0][c];
    for (uint32_t r = 1; r < Cl; ++r) last[c] = max(last[c], s.last[r][c]);
  }
  // The children that entry k goes down to (bit c), and its primitive.
  auto goes_down = [&](uint32_t k, uint32_t &p) {
    if (k >= end) return 0u;
    p = in_pairs[it.pstart + k];
    uint32_t mixed, covered;
    if (cached) {
      mixed = s.mixed[k - block_first]; // the warp wrote it
    } else {
      classify8(p, mixed, covered);
      mixed &= ~covered;
    }
    uint32_t keep = 0;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      if (static_cast<int32_t>(p) > last[c]) keep |= 1u << c;
    return keep & mixed;
  };
  // Walk 2: how many go down, per warp and child (lane c counts child c).
  uint32_t cnt = 0;
  for (uint32_t k0 = first; k0 < end; k0 += kWarp) {
    uint32_t p = 0;
    const uint32_t keep = goes_down(k0 + lane, p);
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      const uint32_t b = __ballot_sync(kFullMask, (keep >> c) & 1u);
      if (lane == c) cnt += __popc(b);
    }
  }
  if (lane < 8) s.warp_count[warp][lane] = cnt;
  __syncthreads();
  if (t < 8) {
    uint32_t run = 0;
    for (uint32_t w = 0; w < kLongWarps; ++w) {
      const uint32_t v = s.warp_count[w][t];
      s.warp_count[w][t] = run;
      run += v;
    }
    share(&s.count[rank][t], run);
  }
  sync_all();
  // Block 0's first lanes take the room and write the children (lane c child c).
  if (rank == 0 && warp == 0) {
    const uint32_t c = lane & 7u;
    uint32_t total = 0;
    for (uint32_t r = 0; r < Cl; ++r) total += s.count[r][c];
    int32_t lf = s.last[0][c];
    for (uint32_t r = 1; r < Cl; ++r) lf = max(lf, s.last[r][c]);
    const int64_t oz = int64_t(2 * cell.z + (c >> 2)) * csize;
    const uint32_t cv = lf >= 0 ? pol.const_value(x.prims[lf], oz, csize) : 0u;
    uint32_t inc = total;
#pragma unroll
    for (uint32_t d = 1; d < 8; d <<= 1) {
      const uint32_t o = __shfl_up_sync(kFullMask, inc, d, 8);
      if (c >= d) inc += o;
    }
    const uint32_t np = __shfl_sync(kFullMask, inc, 7);
    const uint32_t cm =
        __ballot_sync(kFullMask, total != 0 || (Policy::kItemsForConst && lf >= 0)) & 0xffu;
    const uint32_t km = __ballot_sync(kFullMask, lf >= 0) & 0xffu;
    const uint32_t kf = __ballot_sync(kFullMask, lf >= 0 && cv == 1u) & 0xffu;
    const uint32_t ni = __popc(cm);
    uint32_t item_at = 0, pair_at = 0, room = 1;
    if (lane == 0) {
      if (ni) item_at = atomicAdd(&h->item_count[l + 1], ni);
      if (np) pair_at = atomicAdd(&h->pair_count[l + 1], np);
      // this item's own room (an overflow elsewhere fails the edit at the
      // next stage; writing within the buffers meanwhile is harmless)
      if (ni && uint64_t(next_base) + item_at + ni > x.a.item_cap) room = 0;
      if (np && uint64_t(pair_at) + np > x.a.pair_cap) room = 0;
      if (!room) set_status(&h->status, kDevCapacity);
      Item &me = x.a.items[base + wi]; // every thread holds its own copy
      me.child_base = next_base + item_at;
      me.masks = cm | (km << 8) | (kf << 16);
      me.pstart = ni;
    }
    item_at = __shfl_sync(kFullMask, item_at, 0);
    pair_at = __shfl_sync(kFullMask, pair_at, 0);
    room = __shfl_sync(kFullMask, room, 0);
    if (lane < 8 && room) {
      if (lf >= 0) pol.replaced(l, it.old, c);
      if ((cm >> c) & 1u) {
        Item ci{};
        ci.cell = child_cell(it.cell, c);
        ci.old = lf >= 0 ? cv : old_child;
        ci.pstart = pair_at + inc - total;
        ci.pcount = total;
        ci.result = base + wi;
        const uint32_t k = item_at + __popc(cm & ((1u << c) - 1u));
        x.a.items[next_base + k] = ci;
        note_big(x, l + 1, k, total);
      }
    }
    if (lane < 8) share(&s.at[c], pair_at + inc - total);
    if (lane == 0) share(&s.room, room);
  }
  sync_all();
  // Walk 3: each warp appends its part, in order (lane c holds child c's next
  // place).
  if (s.room) {
    uint32_t to = 0;
    if (lane < 8) {
      to = s.at[lane] + s.warp_count[warp][lane];
      if constexpr (Cl > 1)
        for (uint32_t r = 0; r < rank; ++r) to += s.count[r][lane];
    }
    for (uint32_t k0 = first; k0 < end; k0 += kWarp) {
      uint32_t p = 0;
      const uint32_t keep = goes_down(k0 + lane, p);
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
        const uint32_t b = __ballot_sync(kFullMask, (keep >> c) & 1u);
        const uint32_t at = __shfl_sync(kFullMask, to, c);
        if ((keep >> c) & 1u) out_pairs[at + __popc(b & lanemask_lt())] = p;
        if (lane == c) to += __popc(b);
      }
    }
  }
  sync_all(); // the buffers are reused, or the blocks end, only when all are done
}

template <class Policy>
__global__ void __cluster_dims__(kLongCluster, 1, 1) __launch_bounds__(kLongBlock, 1)
    expand_long_kernel(EditCtx x, Policy pol, uint32_t l) {
  namespace cg = cooperative_groups;
  __shared__ LongShared s;
  cg::cluster_group cluster = cg::this_cluster();
  Header *h = x.hdr;
  const uint32_t nbig = min(h->big_count[l], x.a.big_cap / 2u);
  const uint32_t *bigs = big_list(x.a, l);
  const uint32_t base = h->item_off[l];
  const uint32_t next_base = base + h->item_count[l];
  // A failed edit: the blocks of a cluster leave together or not at all (one
  // may see a failure that another has not seen yet).
  const uint32_t failed = edit_failed(h) ? 1u : 0u;
  cluster.sync(); // every block has started: its shared memory may be written
  if (threadIdx.x < kLongCluster)
    *cluster.map_shared_rank(&s.failed[cluster.block_rank()], threadIdx.x) = failed;
  cluster.sync();
  uint32_t any = 0;
  for (uint32_t r = 0; r < kLongCluster; ++r) any |= s.failed[r];
  if (any) {
    cluster.sync(); // no block ends while another may still write to it
    return;
  }
  const uint32_t clusters = gridDim.x / kLongCluster;
  for (uint32_t b = blockIdx.x / kLongCluster; b < nbig; b += clusters)
    if (x.a.items[base + bigs[b]].pcount > kLongList)
      expand_long_item<Policy, kLongCluster>(x, pol, l, bigs[b], base, next_base, s);
  for (uint32_t b = blockIdx.x; b < nbig; b += gridDim.x)
    if (x.a.items[base + bigs[b]].pcount <= kLongList)
      expand_long_item<Policy, 1>(x, pol, l, bigs[b], base, next_base, s);
  cluster.sync(); // (a block's last exchange may still be read by its neighbours)
}

// Blocks of expand_long_kernel for level l: a cluster per item of the level,
// at most a block per SM.
inline uint32_t long_grid(uint32_t l) {
  const uint32_t most = static_cast<uint32_t>(sm_count()) / kLongCluster * kLongCluster;
  return std::max(kLongCluster, level_grid(most, l, 1) / kLongCluster * kLongCluster);
}

} // namespace vx::edit
