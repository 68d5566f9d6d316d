// Hash DAG resident on one B200: hash-consed per-level tables, batched
// primitive edits, the plain per-call voxel-list path, terrain builds,
// queries and a canonical dump.
//
// Storage (one table per level):
//   inner level l < depth: a word pool holding items
//       [child_mask | fill_mask << 8, child refs of child_mask in order]
//     (the reference's canonical item, hash_dag_gpu/detail/node.cuh:266-289)
//     and an open-addressing index of 64-bit slots {tag, ref}; ref = word
//     offset + 2.  An insert reserves an empty slot with the busy marker,
//     appends the item to the pool and publishes {tag, ref} with a release
//     store; readers that meet a busy slot with their tag wait (bounded).
//   leaf level: an open-addressing set of the 64-bit masks themselves;
//     ref = slot + 2.  Masks 0 and ~0 are never stored: refs 0 and 1 are the
//     empty / full subtree of any level (hash_dag_gpu/config.cuh:30-37).
// Structural sharing is by content: two equal subtrees of a level always
// have the same ref, so an edit copies only the paths it changes.
#include "edit_common.cuh"
#include "voxel_b200_device.cuh"
#include "graph.cuh"
#include "plain.cuh"
#include "profile.cuh"
#include "tuning.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <cstdio>
#include <cmath>
#include <new>
#include <type_traits>
#include <vector>

namespace vx::dag {

using namespace vx::edit;

constexpr uint32_t kEmptyRef = 0, kFullRef = 1;
constexpr uint32_t kBusy = 0xffffffffu;
constexpr uint32_t kMaxDepth = 14;
constexpr uint32_t kMaxProbes = 1u << 16;

struct Tables {
  uint32_t depth;
  uint32_t *pool[kMaxDepth];
  uint64_t *index[kMaxDepth];
  uint64_t pool_cap[kMaxDepth];
  uint64_t index_mask[kMaxDepth];
  uint64_t *leaves;
  uint64_t leaf_mask;
  Header *hdr;
};

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 30;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 27;
  x *= 0x94d049bb133111ebull;
  x ^= x >> 31;
  return x;
}

// Hash of an item's n words, fed one word at a time: each word is folded in
// by an xor, a multiply by an odd constant and a rotation (a bijection of
// the state for every word, so items that differ in one word never
// collide), and splitmix64's finaliser spreads the state over all 64 bits.
struct WordHash {
  uint64_t h;
  __device__ __forceinline__ explicit WordHash(uint32_t n) : h(0x243f6a8885a308d3ull ^ n) {}
  __device__ __forceinline__ void add(uint32_t w) {
    const uint64_t x = (h ^ w) * 0x9fb21c651e98df25ull;
    h = (x << 29) | (x >> 35);
  }
  __device__ __forceinline__ uint64_t finish() const { return mix64(h); }
};

__device__ __forceinline__ uint64_t hash_words(const uint32_t *w, uint32_t n) {
  WordHash s(n);
  for (uint32_t i = 0; i < n; ++i) s.add(w[i]);
  return s.finish();
}

// The words of an item as node_find_or_insert sees them: a plain array ...
struct ArrayWords {
  const uint32_t *w;
  uint32_t n;
  __device__ __forceinline__ uint32_t size() const { return n; }
  __device__ __forceinline__ uint64_t hash() const { return hash_words(w, n); }
  __device__ __forceinline__ bool equals(const uint32_t *item) const {
    bool eq = true;
    for (uint32_t i = 0; i < n && eq; ++i) eq = item[i] == w[i];
    return eq;
  }
  __device__ __forceinline__ void write(uint32_t *dst) const {
    for (uint32_t i = 0; i < n; ++i) dst[i] = w[i];
  }
};

// ... or a node's header and its 8 child refs, of which those in the child
// mask follow the header.  Kept in registers: every loop over the children
// unrolls, so no word array goes to local memory.
struct ChildWords {
  uint32_t header; // child_mask | fill_mask << 8
  const uint32_t (&child)[8];
  __device__ __forceinline__ uint32_t size() const { return 1u + __popc(header & 0xffu); }
  __device__ __forceinline__ uint64_t hash() const {
    WordHash s(size());
    s.add(header);
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      if (header & (1u << c)) s.add(child[c]);
    return s.finish();
  }
  __device__ __forceinline__ bool equals(const uint32_t *item) const {
    if (item[0] != header) return false; // equal headers: equal lengths
    bool eq = true;
    uint32_t k = 1;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      if (header & (1u << c)) eq &= item[k++] == child[c];
    return eq;
  }
  __device__ __forceinline__ void write(uint32_t *dst) const {
    dst[0] = header;
    uint32_t k = 1;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      if (header & (1u << c)) dst[k++] = child[c];
  }
};

// ------------------------------------------------------------- reading --

__device__ __forceinline__ uint64_t read_leaf(const Tables &t, uint32_t ref) {
  if (ref == kEmptyRef) return 0ull;
  if (ref == kFullRef) return ~0ull;
  return t.leaves[ref - 2];
}

// Child c of the node `ref` at inner level l (refs 0/1 are uniform subtrees);
// the item format is read by voxel_b200_device.cuh's vx_dag_item_child.
__device__ __forceinline__ uint32_t child_ref(const Tables &t, uint32_t l,
                                              uint32_t ref, uint32_t c) {
  if (ref <= kFullRef) return ref;
  return vx_dag_item_child(t.pool[l] + (ref - 2), c);
}

// ---------------------------------------------------------- hash-consing --

__device__ uint32_t leaf_find_or_insert(const Tables &t, uint64_t mask) {
  uint64_t pos = mix64(mask) & t.leaf_mask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe) {
    const uint64_t v = ld_relaxed_u64(t.leaves + pos);
    if (v == mask) return static_cast<uint32_t>(pos + 2);
    if (v == 0) {
      const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long *>(t.leaves + pos),
                                     0ull, static_cast<unsigned long long>(mask));
      if (old == 0) {
        warp_count_u64(reinterpret_cast<unsigned long long *>(&t.hdr->node_count[t.depth]));
        return static_cast<uint32_t>(pos + 2);
      }
      if (old == mask) return static_cast<uint32_t>(pos + 2);
    }
    pos = (pos + 1) & t.leaf_mask;
  }
  set_status(&t.hdr->status, kDevCapacity);
  return kEmptyRef;
}

// Probes use relaxed loads.  An item found through a published entry is
// read after an acquire fence only when it was inserted by this edit (its
// offset is at or above pool_mark, the pool use when the edit's inserts
// began): items from earlier launches are visible without one, and most
// matches of an edit are such pre-existing subtrees.  Inserts publish with a
// release store.
// WarpCounters: bump the level's pool and node counters with one atomic per
// warp (warp_atomic_add_small), for kernels whose lanes insert side by side;
// a kernel with a few inserting lanes per warp does better with plain ones.
template <class Words, bool WarpCounters = true>
__device__ uint32_t node_find_or_insert(const Tables &t, uint32_t l, const Words &w,
                                        bool *inserted = nullptr) {
  const uint32_t n = w.size();
  const uint64_t h = w.hash();
  const uint32_t tag = static_cast<uint32_t>(h >> 32) | 1u;
  uint64_t *idx = t.index[l];
  uint32_t *pool = t.pool[l];
  const uint32_t mark = t.hdr->pool_mark[l];
  uint64_t pos = h & t.index_mask[l];
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe) {
    uint64_t v = ld_relaxed_u64(idx + pos);
    if (v == 0) {
      const uint64_t claim = (static_cast<uint64_t>(tag) << 32) | kBusy;
      const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long *>(idx + pos),
                                     0ull, static_cast<unsigned long long>(claim));
      if (old == 0) {
        const uint32_t off = WarpCounters ? warp_atomic_add_small(&t.hdr->pool_used[l], n)
                                          : atomicAdd(&t.hdr->pool_used[l], n);
        if (static_cast<uint64_t>(off) + n > t.pool_cap[l]) {
          set_status(&t.hdr->status, kDevCapacity);
          // Leave a dead entry (ref 1 never matches an item) so waiters move on.
          st_release_u64(idx + pos, (static_cast<uint64_t>(tag) << 32) | kFullRef);
          return kEmptyRef;
        }
        w.write(pool + off);
        st_release_u64(idx + pos, (static_cast<uint64_t>(tag) << 32) | (off + 2u));
        if (WarpCounters)
          warp_count_u64(reinterpret_cast<unsigned long long *>(&t.hdr->node_count[l]));
        else
          atomicAdd(reinterpret_cast<unsigned long long *>(&t.hdr->node_count[l]), 1ull);
        if (inserted) *inserted = true;
        return off + 2u;
      }
      v = old;
    }
    if (static_cast<uint32_t>(v >> 32) == tag) {
      uint32_t r = static_cast<uint32_t>(v);
      if (r == kBusy) {
        const uint64_t t0 = global_ns();
        while (r == kBusy) {
          if (global_ns() - t0 > kWaitLimitNs) {
            set_status(&t.hdr->status, kDevTimeout);
            return kEmptyRef;
          }
          __nanosleep(64);
          r = static_cast<uint32_t>(ld_relaxed_u64(idx + pos));
        }
      }
      if (r >= 2u) {
        if (r - 2u >= mark) fence_acq_rel_gpu(); // inserted by this edit
        if (w.equals(pool + (r - 2u))) return r;
      }
    }
    pos = (pos + 1) & t.index_mask[l];
  }
  set_status(&t.hdr->status, kDevCapacity);
  return kEmptyRef;
}

// Canonical ref of a node given its 8 child refs: uniform nodes collapse to
// the sentinels, everything else is hash-consed into level l's table.
template <bool WarpCounters = true>
__device__ uint32_t canon_node(const Tables &t, uint32_t l,
                               const uint32_t (&child)[8]) {
  uint32_t cm = 0, fm = 0;
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    const uint32_t r = child[c];
    if (r == kFullRef) fm |= 1u << c;
    else if (r >= 2u) cm |= 1u << c;
  }
  if (cm == 0) {
    if (fm == 0) return kEmptyRef;
    if (fm == 0xffu) return kFullRef;
  }
  return node_find_or_insert<ChildWords, WarpCounters>(t, l, ChildWords{cm | (fm << 8), child});
}

__device__ __forceinline__ uint32_t canon_leaf(const Tables &t, uint64_t mask) {
  if (mask == 0) return kEmptyRef;
  if (mask == ~0ull) return kFullRef;
  return leaf_find_or_insert(t, mask);
}

// ------------------------------------------------------------ pipeline --

struct Ctx {
  Tables t;
  Arena a;
  const vx_primitive *prims;
  const uint32_t *d_prim_count; // device count (NULL: use host_prim_count)
  uint32_t host_prim_count;
  const uint64_t *sorted_keys; // EditCtx::sorted_keys
};

struct DagTree {
  Tables t;
  static constexpr bool kItemsForConst = false;
  static constexpr uint32_t kValueBits = 0xff00u; // the operation
  __device__ uint32_t child(uint32_t l, uint32_t ref, uint32_t c) const {
    return child_ref(t, l, ref, c);
  }
  __device__ __forceinline__ void children(uint32_t l, uint32_t ref, uint32_t (&out)[8]) const {
    if (ref <= kFullRef) {
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) out[c] = ref;
      return;
    }
    const uint32_t *node = t.pool[l] + (ref - 2u);
    const uint32_t header = node[0];
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      const uint32_t bit = 1u << c;
      out[c] = (header >> (8u + c)) & 1u; // kFullRef or kEmptyRef
      if (header & bit) out[c] = node[1u + __popc(header & (bit - 1u))];
    }
  }
  // Superseded subtrees stay in the tables until vx_dag_compact.
  __device__ void replaced(uint32_t, uint32_t, uint32_t) const {}
  template <bool Terrain>
  __device__ uint32_t classify(const vx_primitive &p, uint32_t world_exp,
                               int64_t ox, int64_t oy, int64_t oz, int64_t n) const {
    return vx::edit::classify<Terrain>(p, world_exp, ox, oy, oz, n);
  }
  __device__ uint32_t const_value(const vx_primitive &p, int64_t, int64_t) const {
    return vx_prim_op(&p) == VX_OP_ADD ? kFullRef : kEmptyRef;
  }
};

// pool_mark = pool_used of every level, before the edit inserts anything.
__global__ void mark_pools_kernel(Tables t) {
  if (threadIdx.x < kMaxDepth) t.hdr->pool_mark[threadIdx.x] = t.hdr->pool_used[threadIdx.x];
}

// Level depth - 1 of a terrain build and of the small cooperative edits:
// evaluate the 8 leaves of every item and hash-cons the item.  Lanes (the
// tuning knob "edit.leafparent_lanes") threads share an item, each evaluating
// children q + Lanes * j of it (q its rank in the group): a small edit has
// fewer items than the chip has lanes, so an item's leaves are spread.
// Batches take leafparent_kernel below.
__device__ void finish_upwards(const Ctx &x, uint32_t parent, uint32_t l);

// Climb: after storing an item's result, finish its ancestors (the single
// cooperative kernel's bottom-up build, without level barriers).
template <bool Terrain, uint32_t Lanes, bool Climb = false>
__device__ __forceinline__ void leafparent_body(Ctx x, Blocks blk) {
  static_assert(Lanes == 2 || Lanes == 4 || Lanes == 8, "2, 4 or 8 lanes per item");
  constexpr uint32_t kPer = 8 / Lanes; // leaves per lane
  constexpr uint32_t kGroupBits = (1u << Lanes) - 1u;
  Header *h = x.t.hdr;
  const uint32_t l = x.t.depth - 1;
  const uint32_t W = h->item_count[l]; // loaded beside the status
  const uint32_t base = h->item_off[l];
  if (edit_failed(h)) return;
  const uint32_t *pairs = x.a.pairs[l & 1u];
  const uint32_t world_exp = x.t.depth + 2;
  const uint32_t lane = lane_id();
  const uint64_t total = static_cast<uint64_t>(W) * Lanes;
  const uint64_t stride = static_cast<uint64_t>(blk.count) * blockDim.x;
  // The item's primitives, Lanes at a time: lane q of the group loads the
  // q-th (one parallel load instead of every lane walking the list).
  __shared__ vx_primitive s_pr[kBlock / Lanes][Lanes];
  const uint32_t grp = threadIdx.x / Lanes;
  const uint32_t gbase = lane & ~(Lanes - 1u);
  const uint32_t gmask = kGroupBits << gbase;
  for (uint64_t g0 = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x - lane;
       g0 < total; g0 += stride) {
    const uint64_t g = g0 + lane;
    const bool have = g < total; // the same for the lanes of a group
    const uint32_t wi = static_cast<uint32_t>(g / Lanes), q = lane & (Lanes - 1u);
    uint32_t result[kPer], old_child[kPer];
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) result[j] = old_child[j] = kEmptyRef;
    Item it{};
    if (have) {
      it = x.a.items[base + wi];
      const Cell cell = unpack_cell(it.cell);
      // Independent loads side by side: the first chunk's pair index and the
      // old node, then its primitive and the old leaves (read speculatively:
      // the kernel is bound by dependent round trips, not by bandwidth).
      int64_t ox[kPer], oy[kPer], oz[kPer];
#pragma unroll
      for (uint32_t j = 0; j < kPer; ++j) {
        const uint32_t c = q + Lanes * j;
        ox[j] = int64_t(2 * cell.x + (c & 1u)) * 4;
        oy[j] = int64_t(2 * cell.y + ((c >> 1) & 1u)) * 4;
        oz[j] = int64_t(2 * cell.z + ((c >> 2) & 1u)) * 4;
      }
      const uint32_t n0 = it.pcount < Lanes ? it.pcount : Lanes;
      const uint32_t pidx = q < n0 ? pairs[it.pstart + q] : 0u;
#pragma unroll
      for (uint32_t j = 0; j < kPer; ++j) old_child[j] = child_ref(x.t, l, it.old, q + Lanes * j);
      vx_primitive first{};
      if (q < n0) first = x.prims[pidx];
      uint64_t old_mask[kPer], mask[kPer];
      bool loaded[kPer], touched[kPer];
#pragma unroll
      for (uint32_t j = 0; j < kPer; ++j) {
        old_mask[j] = read_leaf(x.t, old_child[j]);
        mask[j] = 0;
        loaded[j] = touched[j] = false;
      }
      __syncwarp(gmask); // the group's previous item no longer reads s_pr
      s_pr[grp][q] = first;
      __syncwarp(gmask);
      for (uint32_t k = 0; k < it.pcount; ++k) {
        if (k % Lanes == 0 && k != 0) {
          __syncwarp(gmask); // the previous chunk is no longer read
          if (k + q < it.pcount) s_pr[grp][q] = x.prims[pairs[it.pstart + k + q]];
          __syncwarp(gmask);
        }
        const vx_primitive &pr = s_pr[grp][k % Lanes]; // read in place: fewer registers
        const bool add = vx_prim_op(&pr) == VX_OP_ADD;
#pragma unroll
        for (uint32_t j = 0; j < kPer; ++j) {
          const uint32_t cls = classify<Terrain>(pr, world_exp, ox[j], oy[j], oz[j], 4);
          if (cls == VX_CELL_EMPTY) continue;
          touched[j] = true;
          if (cls == VX_CELL_FULL) {
            mask[j] = add ? ~0ull : 0ull;
            loaded[j] = true;
            continue;
          }
          if (!loaded[j]) {
            mask[j] = old_mask[j];
            loaded[j] = true;
          }
          const uint64_t m = leaf_mask<Terrain>(pr, world_exp, ox[j], oy[j], oz[j]);
          mask[j] = add ? (mask[j] | m) : (mask[j] & ~m);
        }
      }
      // An unchanged mask keeps its canonical ref: no probe of the leaf set.
#pragma unroll
      for (uint32_t j = 0; j < kPer; ++j)
        result[j] = (touched[j] && mask[j] != old_mask[j]) ? canon_leaf(x.t, mask[j])
                                                           : old_child[j];
    }
    // A node whose 8 children all kept their refs is the old node itself
    // (refs are canonical), so its hash-consing is skipped.
    bool mine_changed = false;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) mine_changed |= result[j] != old_child[j];
    const uint32_t changed = __ballot_sync(kFullMask, mine_changed);
    const bool same = ((changed >> gbase) & kGroupBits) == 0u;
    uint32_t child[8];
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j)
#pragma unroll
      for (uint32_t k = 0; k < Lanes; ++k)
        child[k + Lanes * j] = __shfl_sync(kFullMask, result[j], gbase + k);
    // At most 32 / Lanes lanes of a warp insert a node here: plain counters.
    if (have && q == 0) {
      x.a.items[base + wi].result = same ? it.old : canon_node<false>(x.t, l, child);
      if (Climb) finish_upwards(x, it.result, l); // it.result: the parent's index
    }
  }
}

// (eight lanes per item, registers for four blocks: the generator's leaf
// masks need them)
__global__ void __launch_bounds__(kBlock, 4) leafparent_terrain_kernel(Ctx x) {
  leafparent_body<true, 8>(x, launch_blocks());
}

// The same level for edits, a warp taking 32 items at a time: each lane owns
// an item for what is done once per item (its record, its first primitive,
// the old node, the classification of its 8 leaves, the hash-consing of the
// new node), and the leaves that some primitive touches are listed and dealt
// out to the lanes, so that the expensive part, a leaf's mask and its probe,
// runs with full warps.  Nearly every item of a batch has one primitive
// (24.82 M primitives for 24.78 M items at 16,384 spheres in 16384^3), whose
// classification tells which leaves those are; the leaves of an item with
// more are all listed and walk its list.
//
// What bounds it: dependent random reads (item, old node, old leaf, leaf
// probe, node probe, item compare), so 32 items of a warp wait together where
// four lanes per item kept 8 in flight, and the integer and FMA pipes, whose
// work per item is a third of what it was (a touched leaf in four lanes'
// stride idled the others, and hashing ran on one lane in four).  On B200,
// 24.8 M items: 4.58 ms with four lanes per item, 2.65 ms so (2.79 built for
// four resident blocks, 2.61 for six).
// MinBlocks: the knob "edit.leafparent_blocks".  Prefetch (the knob
// "edit.leafparent_prefetch"): the old node of the lane's next item is
// prefetched into L2.
struct WarpLeaves {
  uint32_t ref[8][kWarp];  // [child][item]: old child ref, then the new one
  float4 ball[kWarp];      // of an item with one sphere: the cell's first voxel
                           // relative to its centre, and r^2 + 1
  uint8_t task[8 * kWarp]; // item | child << 5
  uint8_t changed[kWarp];  // the item has a child with a new ref
};

// Climb: as in leafparent_body.
template <bool Prefetch, bool Climb>
__device__ __forceinline__ void leafparent_warps(const Ctx &x, Blocks blk) {
  __shared__ WarpLeaves s_warp[kBlock / kWarp];
  Header *h = x.t.hdr;
  const uint32_t l = x.t.depth - 1;
  const uint32_t W = h->item_count[l]; // loaded beside the status
  const uint32_t base = h->item_off[l];
  if (edit_failed(h)) return;
  const uint32_t *pairs = x.a.pairs[l & 1u];
  const uint32_t lane = lane_id();
  WarpLeaves &s = s_warp[threadIdx.x / kWarp];
  const DagTree tree{x.t};
  const uint32_t stride = blk.count * kBlock;
  for (uint64_t w0 = blk.id * uint64_t(kBlock) + threadIdx.x - lane; w0 < W; w0 += stride) {
    const uint32_t wi = static_cast<uint32_t>(w0) + lane;
    const bool have = w0 + lane < W;
    Item it{};
    uint32_t touched = 0;
    uint32_t info = 0; // covered children | one sphere << 8 | add << 9 | sorted leaf masks << 10
    if (have) {
      it = x.a.items[base + wi];
      uint32_t next_old = kEmptyRef;
      if (Prefetch && w0 + lane + stride < W) next_old = x.a.items[base + wi + stride].old;
      const uint32_t pidx = it.pcount != 0 ? pairs[it.pstart] : 0u;
      uint32_t old_child[8];
      tree.children(l, it.old, old_child);
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) s.ref[c][lane] = old_child[c];
      if (Prefetch && next_old > kFullRef) prefetch_l2(x.t.pool[l] + (next_old - 2u));
      if (x.sorted_keys != nullptr) { // a leaf mask per touched leaf, in child order
        for (uint32_t k = 0; k < it.pcount; ++k)
          touched |= 1u << (static_cast<uint32_t>(x.sorted_keys[it.pstart + k]) & 7u);
        info = 0x400u;
      } else if (it.pcount == 1) {
        const vx_primitive pr = x.prims[pidx];
        const Cell cell = unpack_cell(it.cell);
        if (vx_prim_shape(&pr) == VX_SHAPE_SPHERE && pr.r[0] <= kFloatMaskRadius) {
          sphere_classify_children(pr, cell.x * 8u, cell.y * 8u, cell.z * 8u, 4u, touched, info);
          info |= vx_prim_op(&pr) == VX_OP_ADD ? 0x300u : 0x100u;
          const float r = static_cast<float>(pr.r[0]);
          s.ball[lane] =
              make_float4(static_cast<float>(static_cast<int32_t>(cell.x * 8u) - pr.c[0]),
                          static_cast<float>(static_cast<int32_t>(cell.y * 8u) - pr.c[1]),
                          static_cast<float>(static_cast<int32_t>(cell.z * 8u) - pr.c[2]),
                          r * r + 1.0f);
        } else {
          touched = other_children(x.prims + pidx, it.cell, 4u) & 0xffu;
        }
        const uint32_t cv = tree.const_value(pr, 0, 4);
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) // a leaf that holds the value already (LeftValue)
          if (old_child[c] == cv) touched &= ~(1u << c);
      } else if (it.pcount > 1) {
        touched = 0xffu;
      }
    }
    s.changed[lane] = 0;
    // The touched leaves of all items, listed item by item.
    const uint32_t mine = __popc(touched);
    const uint32_t inc = warp_inclusive_sum(mine);
    const uint32_t tasks = __shfl_sync(kFullMask, inc, kWarp - 1);
    uint32_t at = inc - mine;
    for (uint32_t m = touched; m != 0u; m &= m - 1u)
      s.task[at++] = static_cast<uint8_t>(lane | ((__ffs(m) - 1u) << 5));
    __syncwarp();
    for (uint32_t t0 = 0; t0 < tasks; t0 += kWarp) {
      const bool busy = t0 + lane < tasks;
      const uint32_t task = busy ? s.task[t0 + lane] : 0u;
      const uint32_t src = task & 31u, c = task >> 5;
      const uint32_t src_info = __shfl_sync(kFullMask, info, src);
      const bool one_sphere = (src_info & 0x100u) != 0;
      uint32_t old_ref = kEmptyRef;
      uint64_t old_mask = 0, mask = 0;
      if (busy) {
        old_ref = s.ref[c][src];
        mask = old_mask = read_leaf(x.t, old_ref);
      }
      if (busy && one_sphere) {
        const float4 b = s.ball[src];
        uint64_t m = ~0ull;
        if (((src_info >> c) & 1u) == 0u)
          m = sphere_mask_rows(b.x + ((c & 1u) ? 4.0f : 0.0f), b.y + ((c & 2u) ? 4.0f : 0.0f),
                               b.z + ((c & 4u) ? 4.0f : 0.0f), b.w);
        mask = (src_info & 0x200u) ? (mask | m) : (mask & ~m);
      }
      if (__any_sync(kFullMask, busy && !one_sphere)) { // other shapes, longer lists
        const uint64_t cell_bits = __shfl_sync(kFullMask, it.cell, src);
        const uint32_t pstart = __shfl_sync(kFullMask, it.pstart, src);
        const uint32_t pcount = __shfl_sync(kFullMask, it.pcount, src);
        const uint32_t src_touched = __shfl_sync(kFullMask, touched, src);
        const bool sorted = (src_info & 0x400u) != 0;
        const uint32_t n = one_sphere || !busy ? 0u : (sorted ? 1u : pcount);
        for (uint32_t k = 0; k < n; ++k) {
          const vx_primitive *pr =
              x.prims + (sorted ? pstart + __popc(src_touched & ((1u << c) - 1u)) : pairs[pstart + k]);
          const uint64_t m = sorted ? pr->r[0] | (static_cast<uint64_t>(pr->r[1]) << 32)
                                    : other_leaf_mask(pr, cell_bits, c);
          mask = vx_prim_op(pr) == VX_OP_ADD ? (mask | m) : (mask & ~m);
        }
      }
      // An unchanged mask keeps its canonical ref: no probe of the leaf set.
      if (busy && mask != old_mask) {
        s.ref[c][src] = canon_leaf(x.t, mask);
        s.changed[src] = 1;
      }
    }
    __syncwarp();
    // A node whose 8 children all kept their refs is the old node itself
    // (refs are canonical), so its hash-consing is skipped.
    if (have) {
      uint32_t result = it.old;
      if (s.changed[lane]) {
        uint32_t child[8];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) child[c] = s.ref[c][lane];
        result = canon_node(x.t, l, child);
      }
      x.a.items[base + wi].result = result;
      if (Climb) finish_upwards(x, it.result, l); // it.result: the parent's index
    }
    __syncwarp(); // the next items overwrite the warp's buffers
  }
}

template <int MinBlocks, bool Prefetch>
__global__ void __launch_bounds__(kBlock, MinBlocks) leafparent_kernel(Ctx x) {
  // (the same in every block; sorted leaf masks need no list walks)
  if (x.sorted_keys == nullptr && x.t.hdr->item_count[x.t.depth - 1] <= kWideItems)
    leafparent_body<false, 8>(x, launch_blocks());
  else leafparent_warps<Prefetch, false>(x, launch_blocks());
}

// The rebuilt ref of one item at inner level l from its children's results.
// WarpCounters: the pool and node counters are bumped once per warp, which
// needs every active lane of the warp at the same level (true for the
// level-by-level build, not for climbs, where lanes may be at any level).
// Climb: the children's results come from L2 (other SMs wrote them in this
// launch); the level-by-level build reads them in a later launch.
template <bool WarpCounters = true, bool Climb = false>
__device__ __forceinline__ uint32_t build_item(const Ctx &x, uint32_t l, const Item &it) {
  const uint32_t cm = it.masks & 0xffu, km = (it.masks >> 8) & 0xffu,
                 kf = (it.masks >> 16) & 0xffu;
  uint32_t child[8];
  uint32_t k = 0;
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    const uint32_t bit = 1u << c;
    if (cm & bit) {
      const uint32_t *r = &x.a.items[it.child_base + k++].result;
      child[c] = Climb ? __ldcg(r) : *r;
    } else if (km & bit) {
      child[c] = (kf & bit) ? kFullRef : kEmptyRef;
    }
    else child[c] = child_ref(x.t, l, it.old, c);
  }
  // Every child kept its ref: the node is the old one (refs are canonical).
  bool same = true;
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c)
    if ((cm | km) & (1u << c)) same = same && child[c] == child_ref(x.t, l, it.old, c);
  return same ? it.old : canon_node<WarpCounters>(x.t, l, child);
}

__device__ __forceinline__ void build_body(Ctx x, uint32_t l, Blocks blk) {
  Header *h = x.t.hdr;
  const uint32_t W = h->item_count[l]; // loaded beside the status
  const uint32_t base = h->item_off[l];
  if (edit_failed(h)) return;
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
       i < W; i += static_cast<uint64_t>(blk.count) * blockDim.x)
    x.a.items[base + i].result = build_item(x, l, x.a.items[base + i]);
}

// Bottom-up without level barriers: an item at level l has just stored its
// result; count it off its parent's pending children with one
// acquire-release decrement (its result store is published, and the last
// child sees every sibling's), and when it was the last one rebuild the parent
// and go on up.
__device__ void finish_upwards(const Ctx &x, uint32_t parent, uint32_t l) {
  while (parent != kNoParent) {
    // The parent's own fields were written by its expansion, stages ago:
    // read them while the decrement is in flight (only the children's
    // results need its acquire).
    const Item it = load_item_l2(&x.a.items[parent]);
    if (atomic_sub_acq_rel(&x.a.items[parent].pstart, 1u) != 1u) return;
    --l;
    x.a.items[parent].result = build_item<false, true>(x, l, it);
    parent = it.result; // the grandparent, stored there until now
  }
}

// Items below the leaf-parent level with no child items (every child
// unchanged or uniform) have nothing to wait for: they rebuild at once and
// start their own climb.
__device__ __forceinline__ void rebuild_childless_body(Ctx x, Blocks blk) {
  Header *h = x.t.hdr;
  // Every level's first item, in one round trip.  The levels' items lie one
  // after the other, so one thread takes one item of any level and the climbs
  // run side by side; level by level they had to wait for one another.
  __shared__ uint32_t s_base[kMaxDepth];
  if (threadIdx.x < kMaxDepth) s_base[threadIdx.x] = h->item_off[threadIdx.x];
  if (edit_failed(h)) return; // (its barrier also publishes s_base)
  const uint32_t n = s_base[x.t.depth - 1]; // the first leaf-parent item
  for (uint64_t i = blk.id * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(blk.count) * blockDim.x) {
    const Item it = x.a.items[i];
    if (it.masks & 0xffu) continue;
    uint32_t l = 0;
    while (l + 2 < x.t.depth && s_base[l + 1] <= i) ++l;
    x.a.items[i].result = build_item<false, true>(x, l, it);
    finish_upwards(x, it.result, l);
  }
}

__global__ void __launch_bounds__(kBlock) build_kernel(Ctx x, uint32_t l) {
  build_body(x, l, launch_blocks());
}

__global__ void publish_kernel(Ctx x) {
  Header *h = x.t.hdr;
  if (h->status == kDevOk && h->item_count[0] == 1) h->root = x.a.items[0].result;
}

// A whole edit in one cooperative launch, the stages separated by grid-wide
// barriers instead of kernel boundaries: for small batches, where the ~37
// launches of the level-synchronous pipeline (and their mostly idle grids)
// cost more than the work.  The stages are the kernels' own bodies; long
// primitive lists are expanded block by block with a 256-thread block and a
// 4 KiB classification cache (lists beyond it are classified again).
// Requires every block of the grid to be resident (cudaLaunchCooperativeKernel
// checks it).
constexpr uint32_t kSmallBigCache = 4096;

// From this many leaf-parent items on, a warp takes 32 of them (148 blocks of
// 8 warps hold 37,888 at once): do and undo of 128 primitives 500 -> 347 us,
// of 256 830 -> 490 us on B200.
constexpr uint32_t kWarpLeafItems = 24576;

// With Plain, the edit's input is a voxel list (one op): the first stages
// turn it into leaf-mask primitives (PlainPrep) in place of the sort-based
// preparation of the multi-launch path.
// One block per SM runs it, so it may take up to 255 registers (the
// default cap for 256-thread blocks, 128, made it spill).
template <uint32_t Lanes, bool Plain>
__global__ void __maxnreg__(255) small_edit_kernel(Ctx x, EditCtx e, PlainPrep prep,
                                                            uint32_t *status_out) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const Blocks blk = launch_blocks();
  const DagTree tree{x.t};
  if (Plain) {
    plain_prep_clear(prep, blk);
    grid.sync();
    plain_prep_aggregate(prep, x.t.depth, blk);
    grid.sync();
    plain_prep_fill(prep, blk); // beside init: both need only the final count
  }
  init_body(e, kUseHeaderRoot, blk);
  // pool_mark: nothing is inserted before the leaf-parent level
  if (blk.id == 0 && threadIdx.x < kMaxDepth)
    x.t.hdr->pool_mark[threadIdx.x] = x.t.hdr->pool_used[threadIdx.x];
  grid.sync();
  for (uint32_t l = 0; l + 1 < x.t.depth; ++l) {
    // Short and long lists of level l side by side, one barrier per level:
    // the long ones were listed when level l was emitted (their count is
    // final at the barrier before, the same in every block) and go to the
    // blocks from the last one down, the short ones from block 0 up.
    expand_body<DagTree, false>(e, tree, l, blk);
    if (x.t.hdr->big_count[l] != 0)
      expand_big_body<DagTree, kBlock, kSmallBigCache>(e, tree, l,
                                                   Blocks{blk.count - 1u - blk.id, blk.count});
    grid.sync();
  }
  // The bottom-up build without level barriers: the leaf-parent items and
  // the childless items of the levels above finish their ancestors, each
  // item rebuilt by the last of its children to finish.
  // Many leaf-parent items: 32 a warp; fewer: their leaves over more lanes.
  if (x.t.hdr->item_count[x.t.depth - 1] >= kWarpLeafItems)
    leafparent_warps<false, true>(x, blk);
  else
    leafparent_body<false, Lanes, true>(x, blk);
  // (from the last block down: the leaf-parent items start at the first)
  rebuild_childless_body(x, Blocks{blk.count - 1u - blk.id, blk.count});
  grid.sync();
  if (blk.id == 0 && threadIdx.x == 0) {
    Header *h = x.t.hdr;
    if (h->status == kDevOk && h->item_count[0] == 1) h->root = x.a.items[0].result;
    if (status_out) *status_out = h->status; // the caller's mapped host word
  }
}

__global__ void query_kernel(vx_dag_view v, const vx_voxel *pts, uint32_t n,
                             uint8_t *out) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const vx_voxel p = pts[i];
  out[i] = vx_dag_get_voxel(v, p.x, p.y, p.z);
}

// Rays differ in length by orders of magnitude (a miss of the world, a ray
// along a cave).  Two kernels share a list of rays, 32 at a time:
//
// raycast_kernel, a thread per ray, takes short lists and those groups whose 32
// rays are alike (primary rays of neighbouring pixels): they walk the same
// cells, so the warp stays together, and its blocks are dealt out as others end.
//
// raycast_refill_kernel takes the others.  A thread per ray would leave a warp
// waiting for its longest (5.75 of 32 lanes were active per instruction), so
// a warp takes rays from its share as its lanes' rays end, once kRayRefill
// lanes are idle.  Shares are every so-many-th 32 rays: neighbours in the list
// cost alike.  The cells that a ray's path goes through are kept in a column
// of shared memory per thread.
//
// B200, a 4096^3 DAG, us, a thread per ray / refilling / both kernels as here:
//   1 M rays, half downwards on the terrain, half at random   801 / 590 / 613
//   images of 1024^2 rays from three eyes  393 530 293 / 461 713 305 / 416 548 302
//   images of 2048^2 rays                861 1442 520 / 1221 2079 698 / 900 1490 575
//   65,536 rays                                               209 / 225 / -
//   350,000 such rays, five seeds: 344-494 a thread per ray, 411-491 both kernels
//   440,000: 391-505, 392-480; 700,000: 560-639, 472-524
// Up to kRayFewest rays the longest decide: a thread per ray.  (Refilling at 4,
// 16 and 24 idle lanes, 2 and 8 steps between refills, 4 and 6 blocks per SM:
// 590-800 us for the first.)
constexpr uint32_t kRayRefill = 8, kRaySteps = 4, kRayBlocksPerSm = 5;
constexpr uint32_t kRayFewest = 3u << 17;

// Whether the 32 rays from `first` on are alike: directions within 11.5 degrees
// (cos^2 0.96) of the first one's and origins within a sixteenth of the world
// of its origin; fewer than 32 rays are.  Called by a whole warp.  Rounded
// operations throughout, so that both kernels find the same.
__device__ __forceinline__ bool rays_alike(const vx_ray *rays, uint64_t first, uint32_t n,
                                           float reach) {
  if (first + kWarp > n) return true;
  const vx_ray r = rays[first + lane_id()];
  float dot = 0.0f, mine = 0.0f, lead = 0.0f;
  bool near = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float d0 = __shfl_sync(kFullMask, r.dir[a], 0);
    const float o0 = __shfl_sync(kFullMask, r.origin[a], 0);
    dot = __fadd_rn(dot, __fmul_rn(r.dir[a], d0));
    mine = __fadd_rn(mine, __fmul_rn(r.dir[a], r.dir[a]));
    lead = __fadd_rn(lead, __fmul_rn(d0, d0));
    near = near && fabsf(__fsub_rn(r.origin[a], o0)) <= reach;
  }
  const bool aligned =
      dot > 0.0f && __fmul_rn(dot, dot) >= __fmul_rn(0.96f, __fmul_rn(mine, lead));
  return __all_sync(kFullMask, near && aligned);
}

// All: every ray; otherwise those that rays_alike names.
template <bool All>
__global__ void __launch_bounds__(kBlock)
    raycast_kernel(vx_dag_view v, const vx_ray *rays, uint32_t n, vx_ray_hit *hits, float reach) {
  const uint64_t i = blockIdx.x * uint64_t(kBlock) + threadIdx.x;
  if (i - lane_id() >= n) return;
  if (!All && !rays_alike(rays, i - lane_id(), n, reach)) return;
  if (i < n) hits[i] = vx_dag_raycast(v, rays[i]);
}

__global__ void __launch_bounds__(kBlock, kRayBlocksPerSm)
    raycast_refill_kernel(vx_dag_view v, const vx_ray *rays, uint32_t n, vx_ray_hit *hits,
                          float reach) {
  __shared__ uint32_t s_path[kMaxDepth + 1][kBlock];
  uint32_t *path = &s_path[0][threadIdx.x];
  const uint64_t stride = gridDim.x * uint64_t(kBlock);
  // the warp's current 32 rays and how many of them are taken
  uint64_t first = blockIdx.x * uint64_t(kBlock) + threadIdx.x - lane_id();
  uint32_t taken = 0;
  while (first < n && rays_alike(rays, first, n, reach)) first += stride;
  vx_dag_ray ray;
  uint64_t mine = 0;
  bool active = false;
  for (;;) {
    const uint32_t idle = __ballot_sync(kFullMask, !active);
    if (first < n && __popc(idle) >= kRayRefill) {
      const uint32_t take = taken + __popc(idle & lanemask_lt());
      if (!active && take < kWarp) {
        mine = first + take;
        active = vx_dag_ray_begin(v, rays[mine], ray, path);
        if (!active) hits[mine] = vx_ray_miss();
      }
      taken += __popc(idle);
      if (taken >= kWarp) { // (some idle lanes may wait for the next round)
        taken = 0;
        do first += stride;
        while (first < n && rays_alike(rays, first, n, reach));
      }
    } else if (idle == kFullMask) {
      return; // no ray left
    }
    for (uint32_t k = 0; k < kRaySteps && active; ++k) {
      vx_ray_hit hit;
      if (vx_dag_ray_step(v, ray, path, kBlock, &hit)) {
        hits[mine] = hit;
        active = false;
      }
    }
    __syncwarp();
  }
}

__global__ void read_leaves_kernel(vx_dag_view v, uint32_t lx0, uint32_t ly0, uint32_t lz0,
                                   uint32_t nx, uint32_t ny, uint32_t n, uint64_t *out) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = static_cast<uint32_t>(i % nx), y = static_cast<uint32_t>((i / nx) % ny),
                 z = static_cast<uint32_t>(i / (uint64_t(nx) * ny));
  out[i] = vx_dag_get_leaf(v, lx0 + x, ly0 + y, lz0 + z);
}

// ------------------------------------------------------- plain path prep --

// Leaf keys: the leaf's Morton path, 3 bits per inner level with the root's
// child in the top bits (the reference's make_leaf_key, hash_dag_gpu/detail/
// node.cuh:67-85, widened to 64 bits).  Lists keep them in 32-bit words when
// they fit (depth <= 10, with the bit that marks leaves outside the world),
// which halves the key traffic of the sort: 8.78 M voxels at depth 10 sort in
// 0.32 ms with 32-bit keys against 0.40 ms with 64-bit ones on B200.
constexpr uint32_t kMaxDepthKey32 = 10;

// Bits of v moved to every third bit (v < 2^10 for u32, < 2^21 for u64) and
// back.
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  return (v | (v << 2)) & 0x09249249u;
}
__device__ __forceinline__ uint64_t spread3(uint64_t v) {
  v = (v | (v << 32)) & 0x001f00000000ffffull;
  v = (v | (v << 16)) & 0x001f0000ff0000ffull;
  v = (v | (v << 8)) & 0x100f00f00f00f00full;
  v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
  return (v | (v << 2)) & 0x1249249249249249ull;
}
__device__ __forceinline__ uint32_t compact3(uint64_t v) {
  v &= 0x1249249249249249ull;
  v = (v | (v >> 2)) & 0x10c30c30c30c30c3ull;
  v = (v | (v >> 4)) & 0x100f00f00f00f00full;
  v = (v | (v >> 8)) & 0x001f0000ff0000ffull;
  v = (v | (v >> 16)) & 0x001f00000000ffffull;
  return static_cast<uint32_t>(v | (v >> 32)) & 0x1fffffu;
}
template <class K>
__device__ __forceinline__ K leaf_key(uint32_t lx, uint32_t ly, uint32_t lz) {
  return spread3(K(lx)) | (spread3(K(ly)) << 1) | (spread3(K(lz)) << 2);
}

// Voxel -> (leaf key, bit); voxels outside the world get key 1 << (3 * depth)
// and are dropped.
template <class K>
__global__ void pack_voxels_kernel(const vx_voxel *v, uint32_t n, uint32_t depth, K *keys,
                                   uint32_t *bits) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const vx_voxel p = v[i];
  const uint32_t side_exp = depth + 2;
  const bool outside = ((p.x >> side_exp) | (p.y >> side_exp) | (p.z >> side_exp)) != 0;
  keys[i] = outside ? K(1) << (3 * depth) : leaf_key<K>(p.x >> 2, p.y >> 2, p.z >> 2);
  bits[i] = outside ? 0u : (p.x & 3u) + 4u * (p.y & 3u) + 16u * (p.z & 3u);
}

template <class K>
__global__ void run_flags_kernel(const K *keys, uint32_t n, uint32_t depth, uint32_t *flags) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const bool valid = keys[i] < (K(1) << (3 * depth));
  flags[i] = (valid && (i == 0 || keys[i - 1] != keys[i])) ? 1u : 0u;
}

// Leaf edit command -> (leaf key, command index); leaves outside the world
// get key 1 << (3 * depth) and are dropped.
template <class K>
__global__ void pack_leaf_commands_kernel(const vx_leaf_command *c, uint32_t n, uint32_t depth,
                                          K *keys, uint32_t *index) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const vx_leaf_command cmd = c[i];
  index[i] = static_cast<uint32_t>(i);
  const bool outside =
      ((cmd.leaf_x >> depth) | (cmd.leaf_y >> depth) | (cmd.leaf_z >> depth)) != 0;
  keys[i] = outside ? K(1) << (3 * depth) : leaf_key<K>(cmd.leaf_x, cmd.leaf_y, cmd.leaf_z);
}

// Each run of equal keys ORs its voxel bits (a voxel list) or its commands'
// masks (leaf edit commands, selected by index) into one leaf-mask primitive,
// written with its key by the run's first lane.  A warp takes 32 entries: the
// ORs run over the warp by shuffles, and the run that its last entry belongs
// to is followed past the warp's end 32 entries at a time (by the warp that
// holds its start), so neither dense lists (runs of 64) nor heavy duplicates
// leave one lane walking a run alone: 0.27 -> 0.07 ms for the 8.78 M
// voxels of a sphere of radius 128 on B200.
template <class K, bool Commands>
__global__ void reduce_runs_kernel(const K *keys, const uint32_t *bits,
                                   const vx_leaf_command *cmds, const uint32_t *offsets,
                                   uint32_t n, uint32_t depth, uint32_t op, uint32_t material,
                                   vx_primitive *out, uint64_t *leaf_keys, uint32_t *out_count) {
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  const uint32_t lane = lane_id();
  const uint64_t w0 = i - lane;
  if (w0 >= n) return;
  const K outside = K(1) << (3 * depth);
  auto mask_of = [&](uint64_t j) {
    if constexpr (Commands) {
      const vx_leaf_command &c = cmds[bits[j]];
      return static_cast<uint64_t>(c.voxel_data_low) |
             (static_cast<uint64_t>(c.voxel_data_high) << 32);
    } else {
      return 1ull << bits[j];
    }
  };
  const K key = i < n ? keys[i] : outside;
  K prev = __shfl_up_sync(kFullMask, key, 1);
  if (lane == 0 && w0 != 0) prev = keys[w0 - 1];
  const bool valid = key < outside;
  const bool start = valid && (i == 0 || prev != key);
  uint64_t mask = valid ? mask_of(i) : 0ull;
  const uint32_t starts = __ballot_sync(kFullMask, start);
  // Each run's OR over the warp, in its first lane: run by run while they are
  // few (dense lists have one or two a warp), else by segmented shuffles.
  // (The entries before the first start belong to the warp before.)
  if (__popc(starts) <= 4) {
    for (uint32_t left = starts; left != 0u;) {
      const uint32_t first = __ffs(left) - 1u;
      left &= left - 1u;
      const uint32_t end = left ? __ffs(left) - 1u : kWarp;
      const bool in = valid && lane >= first && lane < end;
      const uint32_t lo = __reduce_or_sync(kFullMask, in ? static_cast<uint32_t>(mask) : 0u);
      const uint32_t hi = __reduce_or_sync(kFullMask, in ? static_cast<uint32_t>(mask >> 32) : 0u);
      if (lane == first) mask = (static_cast<uint64_t>(hi) << 32) | lo;
    }
  } else {
    const uint32_t after = lane == kWarp - 1 ? 0u : starts & ~((2u << lane) - 1u);
    const uint32_t end = after ? __ffs(after) - 1u : kWarp;
#pragma unroll
    for (uint32_t d = 1; d < kWarp; d <<= 1) {
      const uint64_t m = __shfl_down_sync(kFullMask, mask, d);
      if (lane + d < end) mask |= m;
    }
  }
  const K last = __shfl_sync(kFullMask, key, kWarp - 1);
  const uint32_t owner = starts ? 31u - __clz(starts) : 0u;
  if (starts && last < outside && __shfl_sync(kFullMask, key, owner) == last) {
    uint64_t more = 0;
    for (uint64_t j = w0 + kWarp; j < n; j += kWarp) {
      const bool same = j + lane < n && keys[j + lane] == last;
      if (same) more |= mask_of(j + lane);
      if (!__all_sync(kFullMask, same)) break;
    }
    const uint32_t lo = __reduce_or_sync(kFullMask, static_cast<uint32_t>(more));
    const uint32_t hi = __reduce_or_sync(kFullMask, static_cast<uint32_t>(more >> 32));
    if (lane == owner) mask |= (static_cast<uint64_t>(hi) << 32) | lo;
  }
  if (i >= n) return;
  const uint32_t at = start || i == n - 1 ? offsets[i] : 0u;
  if (start) {
    vx_primitive p{};
    p.c[0] = static_cast<int32_t>(compact3(key) * 4u);
    p.c[1] = static_cast<int32_t>(compact3(key >> 1) * 4u);
    p.c[2] = static_cast<int32_t>(compact3(key >> 2) * 4u);
    p.r[0] = static_cast<uint32_t>(mask);
    p.r[1] = static_cast<uint32_t>(mask >> 32);
    p.flags = vx_make_flags(kShapeLeafMask, op, material);
    out[at] = p;
    leaf_keys[at] = key;
  }
  if (i == n - 1) *out_count = at + (start ? 1u : 0u);
}

} // namespace vx::dag

// ================================================================ handle ==

struct vx_dag {
  vx::dag::Tables t{};
  vx::edit::Arena a{};
  uint64_t index_slots[vx::dag::kMaxDepth] = {};
  uint64_t leaf_slots = 0;
  void *arena_mem = nullptr;
  size_t bytes = 0;
  vx_primitive *tmp_prim = nullptr; // one terrain primitive
  uint32_t *host_status = nullptr;  // pinned word for status reads (allocated on first use)
  uint32_t *status_alias = nullptr; // its device address, when mapped at creation
};

namespace vx::dag {

inline uint64_t next_pow2(uint64_t v) {
  uint64_t p = 1;
  while (p < v) p <<= 1;
  return p;
}

// The single cooperative launch of small_edit_kernel, on as many blocks as
// are resident at once (at most the edit.small_blocks_per_sm knob per SM).
// Resident blocks per SM of small_edit_kernel<2 / 4 / 8 lanes, plain or
// not>, queried once (at DAG creation, so never first inside a stream
// capture).
void *small_kernel(int64_t lanes, bool plain) {
  if (plain)
    return lanes == 2   ? reinterpret_cast<void *>(&small_edit_kernel<2, true>)
           : lanes == 4 ? reinterpret_cast<void *>(&small_edit_kernel<4, true>)
                        : reinterpret_cast<void *>(&small_edit_kernel<8, true>);
  return lanes == 2   ? reinterpret_cast<void *>(&small_edit_kernel<2, false>)
         : lanes == 4 ? reinterpret_cast<void *>(&small_edit_kernel<4, false>)
                      : reinterpret_cast<void *>(&small_edit_kernel<8, false>);
}
int g_small_resident[6] = {-1, -1, -1, -1, -1, -1};
inline int small_slot(int64_t lanes, bool plain) {
  return (lanes == 2 ? 0 : (lanes == 4 ? 1 : 2)) + (plain ? 3 : 0);
}
vx_status query_small_residency() {
  const int64_t lanes[3] = {2, 4, 8};
  for (int plain = 0; plain < 2; ++plain)
    for (int i = 0; i < 3; ++i) {
      int &slot = g_small_resident[small_slot(lanes[i], plain != 0)];
      if (slot >= 0) continue;
      int n = 0;
      VX_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, small_kernel(lanes[i], plain != 0), kBlock, 0));
      slot = n;
    }
  return VX_OK;
}

// status_out: a mapped host word the kernel's last act writes the status to.
vx_status run_small(vx_dag *d, Ctx &x, const EditCtx &e, cudaStream_t s,
                    const PlainPrep *prep = nullptr, uint32_t *status_out = nullptr) {
  const int64_t lanes = tune::get(tune::kEditLeafparentLanes);
  void *fn = small_kernel(lanes, prep != nullptr);
  VX_TRY(query_small_residency());
  const int per_sm = g_small_resident[small_slot(lanes, prep != nullptr)];
  const int want = static_cast<int>(tune::get(tune::kEditSmallBlocksPerSm));
  const uint32_t grid = static_cast<uint32_t>(sm_count()) *
                        static_cast<uint32_t>(std::max(1, std::min(per_sm, want)));
  if (per_sm < 1) return VX_ERR_INVALID_VALUE;
  EditCtx ec = e;
  PlainPrep pp = prep ? *prep : PlainPrep{};
  void *args[] = {&x, &ec, &pp, &status_out};
  prof::Scope sc("dag_small_edit", s);
  VX_TRY_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kBlock), args, 0, s));
  (void)d;
  return VX_OK;
}

// Small edits (by the edit.small_max_* knobs) run as one cooperative kernel:
// a batch of primitives by its count, a voxel list or leaf commands (one
// leaf-mask primitive per touched leaf) by its length.
inline bool small_batch(uint32_t n, bool voxel_list) {
  return n <= static_cast<uint32_t>(tune::get(voxel_list ? tune::kEditSmallMaxVoxels
                                                         : tune::kEditSmallMaxPrims));
}

vx_status run_pipeline(vx_dag *d, const vx_primitive *prims,
                       const uint32_t *d_count, uint32_t host_count,
                       cudaStream_t s, bool terrain = false,
                       uint32_t blocks_per_sm = 0 /* 0: the edit.blocks_per_sm knob */,
                       int small = -1 /* -1: by host_count as a primitive batch */,
                       const uint64_t *sorted_keys = nullptr /* EditCtx::sorted_keys */) {
  Ctx x{d->t, d->a, prims, d_count, host_count, nullptr};
  EditCtx e{d->t.hdr, d->a, prims, d_count, host_count, d->t.depth,
            static_cast<uint32_t>(tune::get(tune::kEditBigItem)), nullptr};
  const uint32_t depth = d->t.depth;
  const uint32_t grid = static_cast<uint32_t>(sm_count()) *
                        (blocks_per_sm ? blocks_per_sm
                                       : static_cast<uint32_t>(tune::get(tune::kEditBlocksPerSm)));
  if (!terrain && (small < 0 ? small_batch(host_count, false) : small != 0))
    return run_small(d, x, e, s);
  e.sorted_keys = x.sorted_keys = sorted_keys;
  if (sorted_keys != nullptr) e.big_item = 0xffffffffu; // no list is walked
  {
    prof::Scope sc("dag_init", s);
    init_kernel<<<std::min<uint32_t>(grid, ceil_div(std::max(host_count, 1u), kBlock) + 1),
                  kBlock, 0, s>>>(e, kUseHeaderRoot);
  }
  VX_TRY_CUDA(cudaGetLastError());
  DagTree tree{d->t};
  for (uint32_t l = 0; l + 1 < depth; ++l) {
    const uint32_t lgrid = level_grid(grid, l, kBlock / 8);
    {
      prof::Scope sc("dag_expand", s);
      if (terrain)
        expand_kernel<DagTree, true><<<lgrid, kBlock, 0, s>>>(e, tree, l);
      else if (sorted_keys != nullptr)
        expand_sorted_kernel<DagTree><<<lgrid, kBlock, 0, s>>>(e, tree, l);
      else
        expand_warp_kernel<DagTree>
            <<<expand_grid(grid, l), kBlock, 0, s>>>(e, tree, l);
    }
    VX_TRY_CUDA(cudaGetLastError());
    if (sorted_keys != nullptr || terrain) continue; // no long lists
    {
      prof::Scope sc("dag_expand_big", s);
      expand_long_kernel<DagTree><<<long_grid(l), kLongBlock, 0, s>>>(e, tree, l);
    }
    VX_TRY_CUDA(cudaGetLastError());
  }
  {
    prof::Scope sc("dag_mark_pools", s);
    mark_pools_kernel<<<1, 32, 0, s>>>(d->t);
  }
  VX_TRY_CUDA(cudaGetLastError());
  {
    prof::Scope sc("dag_leafparent", s);
    const int64_t lb = tune::get(tune::kEditLeafparentBlocks);
    const bool prefetch = tune::get(tune::kEditLeafparentPrefetch) != 0;
    auto launch = [&](auto kernel) { kernel<<<grid, kBlock, 0, s>>>(x); };
    if (terrain) launch(leafparent_terrain_kernel);
    else if (lb == 6) launch(prefetch ? leafparent_kernel<6, true> : leafparent_kernel<6, false>);
    else if (lb == 5) launch(prefetch ? leafparent_kernel<5, true> : leafparent_kernel<5, false>);
    else launch(prefetch ? leafparent_kernel<4, true> : leafparent_kernel<4, false>);
  }
  VX_TRY_CUDA(cudaGetLastError());
  for (uint32_t r = depth - 1; r > 0; --r) {
    prof::Scope sc("dag_build", s);
    build_kernel<<<level_grid(grid, r - 1, kBlock), kBlock, 0, s>>>(x, r - 1);
    VX_TRY_CUDA(cudaGetLastError());
  }
  {
    prof::Scope sc("dag_publish", s);
    publish_kernel<<<1, 1, 0, s>>>(x);
  }
  return from_cuda(cudaGetLastError());
}

// A prepared list of `count` voxels or leaf commands: small ones in one
// cooperative launch, the others level by level in key order.
vx_status run_list(vx_dag *d, const vx::plain::Prepared &list, uint32_t count, cudaStream_t s) {
  return run_pipeline(d, list.prims, list.count, count, s, false, 0, small_batch(count, true),
                      list.leaf_keys);
}

// The device status, read through a pinned word (a copy into pageable
// memory goes through a staging buffer); a failed status is cleared.
vx_status read_status(vx_dag *d, cudaStream_t s, bool clear) {
  if (d->host_status == nullptr &&
      cudaHostAlloc(reinterpret_cast<void **>(&d->host_status), sizeof(uint32_t),
                    cudaHostAllocDefault) != cudaSuccess) {
    cudaGetLastError(); // not fatal: read through a stack word instead
    d->host_status = nullptr;
  }
  uint32_t stack_code = 0;
  uint32_t *code = d->host_status ? d->host_status : &stack_code;
  VX_TRY_CUDA(cudaMemcpyAsync(code, &d->t.hdr->status, sizeof(uint32_t),
                              cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  const uint32_t c = *code;
  if (clear && c != kDevOk) {
    VX_TRY_CUDA(cudaMemsetAsync(&d->t.hdr->status, 0, sizeof(uint32_t), s));
    VX_TRY_CUDA(cudaStreamSynchronize(s));
  }
  return status_from_device(c);
}

// The status a small kernel wrote into the mapped host word (set to
// kStatusUnset before the launch): after the kernel there is no copy to
// wait for.  A word the kernel did not write falls back to read_status.
constexpr uint32_t kStatusUnset = 0xffffffffu;
vx_status read_written_status(vx_dag *d, cudaStream_t s) {
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  const uint32_t c = *reinterpret_cast<volatile uint32_t *>(d->host_status);
  if (c == kStatusUnset) return read_status(d, s, true);
  if (c != kDevOk) {
    VX_TRY_CUDA(cudaMemsetAsync(&d->t.hdr->status, 0, sizeof(uint32_t), s));
    VX_TRY_CUDA(cudaStreamSynchronize(s));
  }
  return status_from_device(c);
}

struct PlainLayout {
  uint64_t *keys;
  uint32_t *bits;
  uint32_t *offsets;
  vx_primitive *prims;
  uint32_t *count;
  void *sort_ws;
  size_t sort_ws_bytes;
  void *scan_ws;
  size_t scan_ws_bytes;
};

template <class C> PlainLayout plain_layout(C &c, uint32_t n) {
  PlainLayout p{};
  p.keys = c.template take<uint64_t>(n);
  p.bits = c.template take<uint32_t>(n);
  p.offsets = c.template take<uint32_t>(n);
  p.prims = c.template take<vx_primitive>(n);
  p.count = c.template take<uint32_t>(1);
  p.sort_ws_bytes = vx_sort_workspace_size(n, 8);
  p.sort_ws = c.template take<char>(p.sort_ws_bytes);
  p.scan_ws_bytes = vx_scan_workspace_size(n);
  p.scan_ws = c.template take<char>(p.scan_ws_bytes);
  return p;
}

struct NullCarver {
  size_t offset = 0;
  template <class T> T *take(size_t count) {
    offset = align_up(offset, 256);
    offset += count * sizeof(T);
    return nullptr;
  }
};

} // namespace vx::dag

namespace vx::plain {

size_t workspace_size(uint32_t count) {
  if (count == 0) return 0;
  vx::dag::NullCarver c;
  vx::dag::plain_layout(c, count);
  return c.offset;
}

namespace {

// Packed (leaf key, bit or command index) entries, sorted by key and reduced
// to one leaf-mask primitive per leaf, in key order.
template <class K, class Pack>
vx_status prepare_keys(Pack pack, const vx_leaf_command *cmds, uint32_t count, uint32_t depth,
                       uint32_t op, uint32_t material, void *workspace, Prepared *out,
                       cudaStream_t s) {
  using namespace vx::dag;
  vx::Carver c(workspace);
  const PlainLayout p = plain_layout(c, count);
  const uint32_t blocks = vx::ceil_div(count, kBlock);
  K *keys = reinterpret_cast<K *>(p.keys);
  pack(keys, p.bits, blocks);
  VX_TRY_CUDA(cudaGetLastError());
  if constexpr (sizeof(K) == 4)
    VX_TRY(vx_sort_pairs_u32(keys, p.bits, count, 3 * depth + 1, p.sort_ws, p.sort_ws_bytes, s));
  else
    VX_TRY(vx_sort_pairs_u64(keys, p.bits, count, 3 * depth + 1, p.sort_ws, p.sort_ws_bytes, s));
  {
    vx::prof::Scope sc("plain_run_flags", s);
    run_flags_kernel<K><<<blocks, kBlock, 0, s>>>(keys, count, depth, p.offsets);
  }
  VX_TRY_CUDA(cudaGetLastError());
  VX_TRY(vx_scan_exclusive_sum_u32(p.offsets, count, p.scan_ws, p.scan_ws_bytes, s));
  // The leaves' keys take the place of the sort's scratch (which holds a copy
  // of the 64-bit keys); a list of one entry sorts without scratch, and its
  // own word is read before its leaf's key replaces it.
  uint64_t *leaf_keys = count > 1 ? static_cast<uint64_t *>(p.sort_ws) : p.keys;
  {
    vx::prof::Scope sc("plain_reduce_runs", s);
    if (cmds != nullptr)
      reduce_runs_kernel<K, true><<<blocks, kBlock, 0, s>>>(keys, p.bits, cmds, p.offsets, count,
                                                            depth, op, material, p.prims,
                                                            leaf_keys, p.count);
    else
      reduce_runs_kernel<K, false><<<blocks, kBlock, 0, s>>>(keys, p.bits, nullptr, p.offsets,
                                                             count, depth, op, material, p.prims,
                                                             leaf_keys, p.count);
  }
  VX_TRY_CUDA(cudaGetLastError());
  *out = Prepared{p.prims, p.count, leaf_keys};
  return VX_OK;
}

} // namespace

// Voxel list -> one leaf-mask primitive per touched leaf (op, material),
// written into the workspace.
vx_status prepare(const vx_voxel *edits, uint32_t count, uint32_t depth,
                  uint32_t op, uint32_t material, void *workspace, Prepared *out,
                  cudaStream_t s) {
  using namespace vx::dag;
  auto pack = [&](auto *keys, uint32_t *bits, uint32_t blocks) {
    using K = std::remove_pointer_t<decltype(keys)>;
    vx::prof::Scope sc("plain_pack_voxels", s);
    pack_voxels_kernel<K><<<blocks, kBlock, 0, s>>>(edits, count, depth, keys, bits);
  };
  return depth <= kMaxDepthKey32
             ? prepare_keys<uint32_t>(pack, nullptr, count, depth, op, material, workspace, out, s)
             : prepare_keys<uint64_t>(pack, nullptr, count, depth, op, material, workspace, out, s);
}

// Leaf edit commands -> one leaf-mask primitive per named leaf, the masks of
// commands naming the same leaf OR-merged (the engine's merge_commands).
vx_status prepare_leaf_commands(const vx_leaf_command *cmds, uint32_t count, uint32_t depth,
                                uint32_t op, uint32_t material, void *workspace, Prepared *out,
                                cudaStream_t s) {
  using namespace vx::dag;
  auto pack = [&](auto *keys, uint32_t *index, uint32_t blocks) {
    using K = std::remove_pointer_t<decltype(keys)>;
    vx::prof::Scope sc("plain_pack_leaf_commands", s);
    pack_leaf_commands_kernel<K><<<blocks, kBlock, 0, s>>>(cmds, count, depth, keys, index);
  };
  return depth <= kMaxDepthKey32
             ? prepare_keys<uint32_t>(pack, cmds, count, depth, op, material, workspace, out, s)
             : prepare_keys<uint64_t>(pack, cmds, count, depth, op, material, workspace, out, s);
}

} // namespace vx::plain

using namespace vx::dag;

extern "C" {

vx_status vx_dag_create(const vx_dag_config *cfg, vx_dag **out) {
  if (cfg == nullptr || out == nullptr || cfg->depth < 1 || cfg->depth > kMaxDepth ||
      cfg->max_nodes < 16)
    return VX_ERR_INVALID_VALUE;
  int devs = 0;
  if (cudaGetDeviceCount(&devs) != cudaSuccess || devs == 0) return VX_ERR_NO_DEVICE;
  auto *d = new (std::nothrow) vx_dag;
  if (d == nullptr) return VX_ERR_MEMORY_ALLOCATION;
  d->t.depth = cfg->depth;
  auto fail = [&](cudaError_t e) {
    vx_dag_destroy(d);
    return vx::from_cuda(e);
  };
  cudaError_t e;
  for (uint32_t l = 0; l < cfg->depth; ++l) {
    // Level l holds at most 8^l live nodes, plus superseded ones from earlier
    // edits: every edit copies the path above what it changes, so the small
    // levels fill with garbage first. They keep room for max(2^20,
    // max_nodes / 16) items, which sets how often a long-running editor
    // (the serving loop) has to compact.
    const double live = l < 21 ? std::pow(8.0, static_cast<double>(l)) : 1e30;
    const uint64_t floor_cap = std::max<uint64_t>(1u << 20, cfg->max_nodes / 16);
    const uint64_t cap = std::min<uint64_t>(
        cfg->max_nodes, std::max<uint64_t>(floor_cap, static_cast<uint64_t>(std::min(live * 4, 1e18))));
    d->index_slots[l] = next_pow2(cap * 2);
    d->t.index_mask[l] = d->index_slots[l] - 1;
    d->t.pool_cap[l] = std::min<uint64_t>(cap * 6, 0xfffffff0ull);
    if ((e = cudaMalloc(&d->t.index[l], d->index_slots[l] * 8)) != cudaSuccess) return fail(e);
    if ((e = cudaMalloc(&d->t.pool[l], d->t.pool_cap[l] * 4)) != cudaSuccess) return fail(e);
    d->bytes += d->index_slots[l] * 8 + d->t.pool_cap[l] * 4;
  }
  d->leaf_slots = next_pow2(cfg->max_nodes * 2);
  d->t.leaf_mask = d->leaf_slots - 1;
  if ((e = cudaMalloc(&d->t.leaves, d->leaf_slots * 8)) != cudaSuccess) return fail(e);
  if ((e = cudaMalloc(&d->t.hdr, sizeof(vx::edit::Header))) != cudaSuccess) return fail(e);
  // the status word, mapped so that a small kernel can write it directly
  if (cudaHostAlloc(reinterpret_cast<void **>(&d->host_status), sizeof(uint32_t),
                    cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer(reinterpret_cast<void **>(&d->status_alias), d->host_status,
                               0) != cudaSuccess) {
    cudaGetLastError(); // not fatal: statuses are then copied
    d->status_alias = nullptr;
  }
  if ((e = cudaMalloc(&d->tmp_prim, sizeof(vx_primitive))) != cudaSuccess) return fail(e);
  d->bytes += d->leaf_slots * 8;
  if (vx_status qs = vx::dag::query_small_residency(); qs != VX_OK) {
    vx_dag_destroy(d);
    return qs;
  }
  const uint64_t arena = cfg->arena_bytes ? cfg->arena_bytes : (512ull << 20);
  if ((e = cudaMalloc(&d->arena_mem, arena)) != cudaSuccess) return fail(e);
  d->bytes += arena;
  // Items take 60 % of the arena, the two pair buffers the rest; every
  // sub-buffer starts on a 256-byte boundary.
  const uint64_t big_bytes = std::min<uint64_t>(arena / 64, 4ull << 20) / 256 * 256;
  const uint64_t item_bytes = (arena - big_bytes) / 10 * 6 / 256 * 256;
  d->a.items = static_cast<vx::edit::Item *>(d->arena_mem);
  d->a.item_cap = static_cast<uint32_t>(std::min<uint64_t>(item_bytes / sizeof(vx::edit::Item), 0xffffffffull));
  const uint64_t pair_bytes = (arena - big_bytes - item_bytes) / 2 / 256 * 256;
  d->a.big = reinterpret_cast<uint32_t *>(static_cast<char *>(d->arena_mem) + item_bytes + 2 * pair_bytes);
  d->a.big_cap = static_cast<uint32_t>(big_bytes / 4);
  d->a.pairs[0] = reinterpret_cast<uint32_t *>(static_cast<char *>(d->arena_mem) + item_bytes);
  d->a.pairs[1] = reinterpret_cast<uint32_t *>(static_cast<char *>(d->arena_mem) + item_bytes + pair_bytes);
  d->a.pair_cap = static_cast<uint32_t>(std::min<uint64_t>(pair_bytes / 4, 0xffffffffull));
  const vx_status st = vx_dag_reset(d, nullptr);
  if (st != VX_OK) {
    vx_dag_destroy(d);
    return st;
  }
  if ((e = cudaStreamSynchronize(nullptr)) != cudaSuccess) return fail(e);
  *out = d;
  return VX_OK;
}

vx_status vx_dag_destroy(vx_dag *d) {
  if (d == nullptr) return VX_ERR_INVALID_VALUE;
  for (uint32_t l = 0; l < kMaxDepth; ++l) {
    cudaFree(d->t.index[l]);
    cudaFree(d->t.pool[l]);
  }
  cudaFree(d->t.leaves);
  cudaFree(d->t.hdr);
  cudaFree(d->arena_mem);
  cudaFree(d->tmp_prim);
  if (d->host_status) cudaFreeHost(d->host_status);
  delete d;
  return VX_OK;
}

vx_status vx_dag_reset(vx_dag *d, vx_stream stream) {
  if (d == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (uint32_t l = 0; l < d->t.depth; ++l)
    VX_TRY_CUDA(cudaMemsetAsync(d->t.index[l], 0, d->index_slots[l] * 8, s));
  VX_TRY_CUDA(cudaMemsetAsync(d->t.leaves, 0, d->leaf_slots * 8, s));
  VX_TRY_CUDA(cudaMemsetAsync(d->t.hdr, 0, sizeof(vx::edit::Header), s));
  return VX_OK;
}

uint32_t vx_dag_depth(const vx_dag *d) { return d ? d->t.depth : 0; }

size_t vx_dag_voxel_workspace_size(uint32_t count) {
  return vx::plain::workspace_size(count);
}

vx_status vx_dag_apply_voxels(vx_dag *d, const vx_voxel *edits, uint32_t count,
                              uint32_t op, void *workspace,
                              size_t workspace_bytes, vx_stream stream) {
  if (d == nullptr || (edits == nullptr && count != 0) || op > 1)
    return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  if (workspace == nullptr || workspace_bytes < vx_dag_voxel_workspace_size(count))
    return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PlainPrep prep;
  if (small_batch(count, true) &&
      plain_prep_layout(workspace, workspace_bytes, edits, count, op, 0, &prep)) {
    // one cooperative launch: voxels -> leaf masks -> the edit
    Ctx x{d->t, d->a, prep.prims, prep.nprims, count, nullptr};
    const EditCtx e{d->t.hdr, d->a, prep.prims, prep.nprims, count, d->t.depth,
                    static_cast<uint32_t>(vx::tune::get(vx::tune::kEditBigItem)), nullptr};
    if (d->status_alias == nullptr) {
      VX_TRY(run_small(d, x, e, s, &prep));
      return read_status(d, s, true);
    }
    *reinterpret_cast<volatile uint32_t *>(d->host_status) = kStatusUnset;
    VX_TRY(run_small(d, x, e, s, &prep, d->status_alias));
    return read_written_status(d, s);
  }
  vx::plain::Prepared list;
  VX_TRY(vx::plain::prepare(edits, count, d->t.depth, op, 0, workspace, &list, s));
  VX_TRY(run_list(d, list, count, s));
  return read_status(d, s, true);
}

size_t vx_leaf_command_workspace_size(uint32_t count) { return vx::plain::workspace_size(count); }

vx_status vx_dag_apply_leaf_commands(vx_dag *d, const vx_leaf_command *cmds, uint32_t count,
                                     uint32_t op, void *workspace, size_t workspace_bytes,
                                     vx_stream stream) {
  if (d == nullptr || (cmds == nullptr && count != 0) || op > 1) return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  if (workspace == nullptr || workspace_bytes < vx_leaf_command_workspace_size(count))
    return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::plain::Prepared list;
  VX_TRY(vx::plain::prepare_leaf_commands(cmds, count, d->t.depth, op, 0, workspace, &list, s));
  VX_TRY(run_list(d, list, count, s));
  return read_status(d, s, true);
}

vx_status vx_dag_apply_primitives(vx_dag *d, const vx_primitive *prims,
                                  uint32_t count, vx_stream stream) {
  if (d == nullptr || (prims == nullptr && count != 0)) return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  return run_pipeline(d, prims, nullptr, count, static_cast<cudaStream_t>(stream));
}

vx_status vx_dag_graph_primitives(vx_dag *d, const vx_primitive *prims,
                                  const uint32_t *device_count, uint32_t capacity,
                                  vx_graph **out) {
  if (d == nullptr || out == nullptr || prims == nullptr || capacity == 0)
    return VX_ERR_INVALID_VALUE;
  return vx::graph::capture(
      [&](cudaStream_t s) { return run_pipeline(d, prims, device_count, capacity, s); }, out);
}

} // extern "C"

namespace vx::dag {
vx_status graph_primitives_grid(vx_dag *d, const vx_primitive *prims, const uint32_t *d_count,
                                uint32_t capacity, uint32_t blocks_per_sm, vx_graph **out) {
  if (d == nullptr || out == nullptr || prims == nullptr || capacity == 0)
    return VX_ERR_INVALID_VALUE;
  return vx::graph::capture(
      [&](cudaStream_t s) {
        return run_pipeline(d, prims, d_count, capacity, s, false, blocks_per_sm);
      },
      out);
}
} // namespace vx::dag

extern "C" {

vx_status vx_dag_graph_voxels(vx_dag *d, const vx_voxel *edits, uint32_t count, uint32_t op,
                              void *workspace, size_t workspace_bytes, vx_graph **out) {
  if (d == nullptr || out == nullptr || edits == nullptr || count == 0 || op > 1)
    return VX_ERR_INVALID_VALUE;
  if (workspace == nullptr || workspace_bytes < vx_dag_voxel_workspace_size(count))
    return VX_ERR_INVALID_VALUE;
  return vx::graph::capture(
      [&](cudaStream_t s) {
        vx::plain::Prepared list;
        VX_TRY(vx::plain::prepare(edits, count, d->t.depth, op, 0, workspace, &list, s));
        return run_list(d, list, count, s);
      },
      out);
}

vx_status vx_dag_status(vx_dag *d, vx_stream stream) {
  if (d == nullptr) return VX_ERR_INVALID_VALUE;
  return read_status(d, static_cast<cudaStream_t>(stream), true);
}

vx_status vx_dag_build_terrain(vx_dag *d, const vx_terrain *terrain,
                               vx_stream stream) {
  if (d == nullptr || terrain == nullptr || terrain->scale == 0) return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx_primitive p{};
  p.c[0] = static_cast<int32_t>(terrain->seed);
  p.c[1] = static_cast<int32_t>(terrain->scale);
  p.c[2] = static_cast<int32_t>(terrain->caves);
  p.flags = vx_make_flags(vx::edit::kShapeTerrain, VX_OP_ADD, 0);
  VX_TRY(vx_dag_reset(d, stream));
  VX_TRY_CUDA(cudaMemcpyAsync(d->tmp_prim, &p, sizeof(p), cudaMemcpyHostToDevice, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  return run_pipeline(d, d->tmp_prim, nullptr, 1, s, true);
}

vx_status vx_dag_query(const vx_dag *d, const vx_voxel *pts, uint32_t count,
                       uint8_t *out, vx_stream stream) {
  if (d == nullptr || ((pts == nullptr || out == nullptr) && count != 0))
    return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::prof::Scope sc("dag_query", s);
  vx_dag_view view;
  VX_TRY(vx_dag_device_view(d, &view));
  query_kernel<<<vx::ceil_div(count, kBlock), kBlock, 0, s>>>(view, pts, count, out);
  return vx::from_cuda(cudaGetLastError());
}

vx_status vx_dag_raycast(const vx_dag *d, const vx_ray *rays, uint32_t count,
                         vx_ray_hit *hits, vx_stream stream) {
  if (d == nullptr || ((rays == nullptr || hits == nullptr) && count != 0))
    return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::prof::Scope sc("dag_raycast", s);
  vx_dag_view view;
  VX_TRY(vx_dag_device_view(d, &view));
  const uint32_t blocks = vx::ceil_div(count, kBlock);
  const float reach = static_cast<float>(4u << view.depth) / 16.0f;
  if (count <= kRayFewest) {
    raycast_kernel<true><<<blocks, kBlock, 0, s>>>(view, rays, count, hits, reach);
    return vx::from_cuda(cudaGetLastError());
  }
  raycast_kernel<false><<<blocks, kBlock, 0, s>>>(view, rays, count, hits, reach);
  VX_TRY_CUDA(cudaGetLastError());
  raycast_refill_kernel<<<std::min(blocks, static_cast<uint32_t>(vx::sm_count()) * kRayBlocksPerSm),
                          kBlock, 0, s>>>(view, rays, count, hits, reach);
  return vx::from_cuda(cudaGetLastError());
}

vx_status vx_dag_read_leaves(const vx_dag *d, uint32_t lx0, uint32_t ly0, uint32_t lz0,
                             uint32_t nx, uint32_t ny, uint32_t nz, uint64_t *out,
                             vx_stream stream) {
  const uint64_t n = uint64_t(nx) * ny * nz;
  if (d == nullptr || (out == nullptr && n != 0) || n >= (1ull << 32)) return VX_ERR_INVALID_VALUE;
  if (n == 0) return VX_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::prof::Scope sc("dag_read_leaves", s);
  vx_dag_view view;
  VX_TRY(vx_dag_device_view(d, &view));
  read_leaves_kernel<<<vx::ceil_div(static_cast<uint32_t>(n), kBlock), kBlock, 0, s>>>(
      view, lx0, ly0, lz0, nx, ny, static_cast<uint32_t>(n), out);
  return vx::from_cuda(cudaGetLastError());
}

vx_status vx_dag_device_view(const vx_dag *d, vx_dag_view *out) {
  if (d == nullptr || out == nullptr) return VX_ERR_INVALID_VALUE;
  *out = vx_dag_view{};
  out->depth = d->t.depth;
  out->root = &d->t.hdr->root;
  for (uint32_t l = 0; l < d->t.depth; ++l) out->pool[l] = d->t.pool[l];
  out->leaves = d->t.leaves;
  return VX_OK;
}

vx_status vx_dag_get_stats(const vx_dag *d, vx_dag_stats *st, vx_stream stream) {
  if (d == nullptr || st == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::edit::Header h;
  VX_TRY_CUDA(cudaMemcpyAsync(&h, d->t.hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  *st = vx_dag_stats{};
  for (uint32_t l = 0; l <= d->t.depth && l < 16; ++l) {
    st->nodes_per_level[l] = h.node_count[l];
    st->words_per_level[l] = l < d->t.depth ? h.pool_used[l] : 2 * h.node_count[l];
  }
  for (uint32_t l = 0; l < 16; ++l) {
    st->items_per_level[l] = h.item_count[l];
    st->pairs_per_level[l] = h.pair_count[l];
  }
  st->bytes_reserved = d->bytes;
  st->root = h.root;
  st->status = h.status;
  return VX_OK;
}

vx_status vx_dag_export_canonical(const vx_dag *d, uint32_t *host_root,
                                  uint64_t *host_counts, uint32_t *host_nodes,
                                  uint64_t nodes_capacity_words,
                                  uint64_t *host_leaves,
                                  uint64_t leaves_capacity, vx_stream stream) {
  return vx_dag_export_canonical_at(d, 0xffffffffu, host_root, host_counts, host_nodes,
                                    nodes_capacity_words, host_leaves, leaves_capacity,
                                    stream);
}

vx_status vx_dag_export_canonical_at(const vx_dag *d, uint32_t root, uint32_t *host_root,
                                     uint64_t *host_counts, uint32_t *host_nodes,
                                     uint64_t nodes_capacity_words,
                                     uint64_t *host_leaves, uint64_t leaves_capacity,
                                     vx_stream stream) {
  if (d == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t D = d->t.depth;
  vx::edit::Header h;
  VX_TRY_CUDA(cudaMemcpyAsync(&h, d->t.hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  if (root != 0xffffffffu) h.root = root;
  std::vector<std::vector<uint32_t>> pools(D);
  for (uint32_t l = 0; l < D; ++l) {
    const uint64_t used = std::min<uint64_t>(h.pool_used[l], d->t.pool_cap[l]);
    pools[l].resize(used);
    if (used)
      VX_TRY_CUDA(cudaMemcpyAsync(pools[l].data(), d->t.pool[l], used * 4,
                                  cudaMemcpyDeviceToHost, s));
  }
  std::vector<uint64_t> leaves(d->leaf_slots);
  VX_TRY_CUDA(cudaMemcpyAsync(leaves.data(), d->t.leaves, d->leaf_slots * 8,
                              cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  // DFS first-visit numbering per level (children 0..7).
  std::vector<std::vector<uint32_t>> out_nodes(D);
  std::vector<uint64_t> out_leaves;
  std::vector<std::vector<int64_t>> ids(D + 1);
  for (uint32_t l = 0; l < D; ++l) ids[l].assign(pools[l].size() + 2, -1);
  std::vector<int64_t> leaf_ids(d->leaf_slots + 2, -1);
  // iterative DFS with an explicit stack of (level, ref, next child)
  struct Frame {
    uint32_t l, ref, c, id;
    uint32_t rec[10];
  };
  auto visit_leaf = [&](uint32_t ref) -> uint32_t {
    if (leaf_ids[ref] < 0) {
      leaf_ids[ref] = static_cast<int64_t>(out_leaves.size());
      out_leaves.push_back(leaves[ref - 2]);
    }
    return static_cast<uint32_t>(leaf_ids[ref]) + 2;
  };
  uint32_t root_id = h.root;
  if (h.root >= 2) {
    if (D == 0) return VX_ERR_INVALID_VALUE;
    std::vector<Frame> st;
    auto open = [&](uint32_t l, uint32_t ref) {
      Frame f{};
      f.l = l;
      f.ref = ref;
      f.c = 0;
      f.id = static_cast<uint32_t>(out_nodes[l].size() / 10);
      ids[l][ref] = f.id;
      out_nodes[l].resize(out_nodes[l].size() + 10, 0);
      st.push_back(f);
    };
    open(0, h.root);
    root_id = 2;
    while (!st.empty()) {
      Frame &f = st.back();
      if (f.c == 8) {
        for (uint32_t w = 0; w < 10; ++w) out_nodes[f.l][f.id * 10 + w] = f.rec[w];
        const uint32_t id = f.id, l = f.l;
        st.pop_back();
        if (!st.empty()) {
          Frame &p = st.back();
          p.rec[2 + p.c] = id + 2;
          p.rec[0] |= 1u << p.c;
          ++p.c;
        }
        (void)l;
        continue;
      }
      const uint32_t *item = pools[f.l].data() + (f.ref - 2);
      const uint32_t cm = item[0] & 0xffu, fm = (item[0] >> 8) & 0xffu;
      const uint32_t bit = 1u << f.c;
      if (cm & bit) {
        const uint32_t child = item[1 + __builtin_popcount(cm & (bit - 1u))];
        if (f.l + 1 == D) {
          f.rec[2 + f.c] = visit_leaf(child);
          f.rec[0] |= bit;
          ++f.c;
        } else if (ids[f.l + 1][child] >= 0) {
          f.rec[2 + f.c] = static_cast<uint32_t>(ids[f.l + 1][child]) + 2;
          f.rec[0] |= bit;
          ++f.c;
        } else {
          open(f.l + 1, child); // completes when popped
        }
      } else {
        if (fm & bit) {
          f.rec[2 + f.c] = 1;
          f.rec[1] |= bit;
        }
        ++f.c;
      }
    }
  }
  if (host_root) *host_root = root_id;
  uint64_t words = 0;
  for (uint32_t l = 0; l < D; ++l) {
    if (host_counts) host_counts[l] = out_nodes[l].size() / 10;
    words += out_nodes[l].size();
  }
  if (host_counts) host_counts[D] = out_leaves.size();
  if (host_nodes) {
    if (words > nodes_capacity_words) return VX_ERR_INVALID_VALUE;
    uint64_t o = 0;
    for (uint32_t l = 0; l < D; ++l)
      for (uint32_t w : out_nodes[l]) host_nodes[o++] = w;
  }
  if (host_leaves) {
    if (out_leaves.size() > leaves_capacity) return VX_ERR_INVALID_VALUE;
    std::copy(out_leaves.begin(), out_leaves.end(), host_leaves);
  }
  return VX_OK;
}

} // extern "C"

// ============================================================ snapshots ==

extern "C" {

// Copy the whole table state (roots, counters, indexes, pools, leaves) of src
// into dst; both must have been created with the same configuration.
vx_status vx_dag_copy(vx_dag *dst, const vx_dag *src, vx_stream stream) {
  if (dst == nullptr || src == nullptr || dst->t.depth != src->t.depth ||
      dst->leaf_slots != src->leaf_slots)
    return VX_ERR_INVALID_VALUE;
  for (uint32_t l = 0; l < src->t.depth; ++l)
    if (dst->index_slots[l] != src->index_slots[l] ||
        dst->t.pool_cap[l] != src->t.pool_cap[l])
      return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  vx::edit::Header h;
  VX_TRY_CUDA(cudaMemcpyAsync(&h, src->t.hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  for (uint32_t l = 0; l < src->t.depth; ++l) {
    VX_TRY_CUDA(cudaMemcpyAsync(dst->t.index[l], src->t.index[l],
                                src->index_slots[l] * 8, cudaMemcpyDeviceToDevice, s));
    const uint64_t used = std::min<uint64_t>(h.pool_used[l], src->t.pool_cap[l]);
    if (used)
      VX_TRY_CUDA(cudaMemcpyAsync(dst->t.pool[l], src->t.pool[l], used * 4,
                                  cudaMemcpyDeviceToDevice, s));
  }
  VX_TRY_CUDA(cudaMemcpyAsync(dst->t.leaves, src->t.leaves, src->leaf_slots * 8,
                              cudaMemcpyDeviceToDevice, s));
  VX_TRY_CUDA(cudaMemcpyAsync(dst->t.hdr, src->t.hdr, sizeof(vx::edit::Header),
                              cudaMemcpyDeviceToDevice, s));
  return VX_OK;
}

} // extern "C"

// ============================================================ compaction ==
//
// Edits are copy-on-write: every changed node gets a new item and the items
// it replaced stay in the tables until compaction (the reference CPU DAG's
// collect_garbage, svt/hash_dag.hpp:133-191).  Compaction marks the nodes
// reachable from the root level by level, stages their items, clears every
// table and hash-conses the live items back bottom-up, remapping child refs
// through sorted (old ref -> new ref) arrays of the level below.  It is a
// maintenance call: it synchronises, and its temporaries live in the DAG's
// edit arena (VX_ERR_CAPACITY if the arena cannot hold them).

namespace vx::dag {

// Compaction.  Every level l gets a mark bitmap over its old ref space (ref
// - 2 = pool word offset, or leaf slot) and, after an exclusive scan of the
// bitmap words' popcounts, a rank for every live ref: the live refs of a
// level, listed in ascending order, are ranks 0..live-1, and the new ref of
// an old one is new_refs[rank(old)].  Nothing is sized on the host except by
// upper bounds, so the whole pass is stream-ordered.
struct LevelMarks {
  uint32_t *bits;   // mark bitmap word w at bits[2w]; bits[2w + 1] holds prefix[w]
                    // once ranked, so that a rank costs one 8-byte load
  uint32_t *prefix; // exclusive prefix of popcount(bits[2w]) (the scan's array)
  uint32_t *refs;   // live old refs in ascending order (rank order)
  uint32_t *new_refs;
  uint32_t *live;   // device count of live refs
  uint64_t words;   // bitmap words
  uint32_t cap;     // capacity of refs / new_refs
};

__device__ __forceinline__ uint32_t rank_of(const LevelMarks &m, uint32_t ref) {
  const uint32_t b = ref - 2u;
  const uint2 w = reinterpret_cast<const uint2 *>(m.bits)[b >> 5]; // {bits, prefix}
  return w.y + __popc(w.x & ((1u << (b & 31u)) - 1u));
}

// Marks the children of level l's live items in level l+1's bitmap.
__global__ void mark_children_kernel(Tables t, uint32_t l, LevelMarks m, LevelMarks next) {
  const uint32_t n = *m.live;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t *item = t.pool[l] + (m.refs[i] - 2);
    const uint32_t cm = item[0] & 0xffu;
    for (uint32_t k = 0; k < static_cast<uint32_t>(__popc(cm)); ++k) {
      const uint32_t b = item[1 + k] - 2u;
      const uint32_t bit = 1u << (b & 31u);
      uint32_t *word = next.bits + 2u * (b >> 5);
      if (!(ld_relaxed_u32(word) & bit)) atomicOr(word, bit);
    }
  }
}

__global__ void popcount_kernel(LevelMarks m) {
  for (uint64_t w = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; w < m.words;
       w += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    m.prefix[w] = __popc(m.bits[2 * w]);
}

// After the scan: the live count and the rank-ordered list of live refs.
__global__ void list_kernel(Tables t, LevelMarks m) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint64_t first = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (first == 0) {
    const uint64_t last = m.words - 1;
    const uint32_t total = m.prefix[last] + __popc(m.bits[2 * last]);
    if (total > m.cap) set_status(&t.hdr->status, kDevCapacity);
    *m.live = min(total, m.cap);
  }
  for (uint64_t w = first; w < m.words; w += stride) {
    uint32_t bits = m.bits[2 * w];
    uint32_t at = m.prefix[w];
    m.bits[2 * w + 1] = at; // beside the bitmap word, for rank_of
    while (bits) {
      const uint32_t b = __ffs(bits) - 1u;
      bits &= bits - 1u;
      if (at < m.cap) m.refs[at] = static_cast<uint32_t>(w * 32u + b + 2u);
      ++at;
    }
  }
}

__global__ void stage_kernel(Tables t, uint32_t l, LevelMarks m,
                             uint32_t *staged /* 9 words per item */, uint64_t *leaf_masks) {
  const uint32_t n = *m.live;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    if (l == t.depth) {
      leaf_masks[i] = t.leaves[m.refs[i] - 2];
      continue;
    }
    const uint32_t *item = t.pool[l] + (m.refs[i] - 2);
    const uint32_t w = 1 + __popc(item[0] & 0xffu);
    for (uint32_t k = 0; k < 9; ++k) staged[i * 9 + k] = k < w ? item[k] : 0u;
  }
}

// Re-insertion.  The live items of a level are distinct by content (the
// tables hash-cons them) and stay distinct after their children are renamed
// (renaming is injective), so an item needs no lookup: its pool offset is the
// exclusive scan of the items' word counts and its index entry takes the
// first empty slot of its probe sequence.  No shared counter is touched per
// item; the level's counts are written once at the end.
// Unique inserts (the item is known not to be in the table): the leaf takes
// the first empty slot of its probe sequence; the node is written at its
// pool offset and its index entry takes the first empty slot.
__device__ uint32_t unique_insert_leaf(const Tables &t, uint64_t mask) {
  uint64_t pos = mix64(mask) & t.leaf_mask;
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe) {
    if (ld_relaxed_u64(t.leaves + pos) == 0 &&
        atomicCAS(reinterpret_cast<unsigned long long *>(t.leaves + pos), 0ull,
                  static_cast<unsigned long long>(mask)) == 0ull)
      return static_cast<uint32_t>(pos + 2);
    pos = (pos + 1) & t.leaf_mask;
  }
  set_status(&t.hdr->status, kDevCapacity);
  return kEmptyRef;
}

__device__ uint32_t unique_insert_node(const Tables &t, uint32_t l, const uint32_t *w,
                                       uint32_t n, uint32_t off) {
  if (static_cast<uint64_t>(off) + n > t.pool_cap[l]) {
    set_status(&t.hdr->status, kDevCapacity);
    return kEmptyRef;
  }
  uint32_t *dst = t.pool[l] + off;
  for (uint32_t j = 0; j < n; ++j) dst[j] = w[j];
  const uint64_t h = hash_words(w, n);
  const uint64_t entry =
      (static_cast<uint64_t>(static_cast<uint32_t>(h >> 32) | 1u) << 32) | (off + 2u);
  uint64_t *idx = t.index[l];
  uint64_t pos = h & t.index_mask[l];
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe) {
    if (ld_relaxed_u64(idx + pos) == 0 &&
        atomicCAS(reinterpret_cast<unsigned long long *>(idx + pos), 0ull,
                  static_cast<unsigned long long>(entry)) == 0ull)
      return off + 2u;
    pos = (pos + 1) & t.index_mask[l];
  }
  set_status(&t.hdr->status, kDevCapacity);
  return off + 2u;
}

__global__ void reinsert_leaves_kernel(Tables t, LevelMarks m, const uint64_t *masks) {
  const uint32_t n = *m.live;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    m.new_refs[i] = unique_insert_leaf(t, masks[i]);
}

__global__ void item_words_kernel(LevelMarks m, const uint32_t *staged, uint32_t *words) {
  const uint32_t n = *m.live;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    words[i] = 1u + __popc(staged[i * 9] & 0xffu);
}

__global__ void reinsert_nodes_kernel(Tables t, uint32_t l, LevelMarks m, LevelMarks child,
                                      const uint32_t *staged, const uint32_t *offsets) {
  const uint32_t n = *m.live;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint32_t w[9];
    w[0] = staged[i * 9];
    const uint32_t k = __popc(w[0] & 0xffu);
    for (uint32_t j = 0; j < k; ++j) w[1 + j] = child.new_refs[rank_of(child, staged[i * 9 + 1 + j])];
    m.new_refs[i] = unique_insert_node(t, l, w, 1 + k, offsets[i]);
  }
}

// ---- import of a canonical dump (records of 10 words per inner node:
// [child_mask, fill_mask, child ids x 8], id k + 2 = node k of the next
// level; leaves as u64 masks).  Canonical nodes are distinct per level, so
// the unique inserts above apply; child ids are checked against the next
// level's count (a malformed dump raises kDevInvalid, never an out-of-range
// read).

__global__ void import_leaves_kernel(Tables t, const uint64_t *masks, uint32_t n,
                                     uint32_t *new_refs) {
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t m = masks[i];
    if (m == 0 || m == ~0ull) {
      set_status(&t.hdr->status, kDevInvalid);
      new_refs[i] = kEmptyRef;
      continue;
    }
    new_refs[i] = unique_insert_leaf(t, m);
  }
}

__global__ void import_words_kernel(const uint32_t *rec, uint32_t n, uint32_t *words) {
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
    words[i] = 1u + __popc(rec[i * 10] & 0xffu);
}

__global__ void import_nodes_kernel(Tables t, uint32_t l, const uint32_t *rec, uint32_t n,
                                    const uint32_t *child_refs, uint32_t child_count,
                                    const uint32_t *offsets, uint32_t *new_refs) {
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t *r = rec + i * 10;
    const uint32_t cm = r[0] & 0xffu, fm = r[1] & 0xffu;
    uint32_t w[9];
    w[0] = cm | (fm << 8);
    uint32_t k = 0;
    bool ok = (cm & fm) == 0 && (cm != 0 || (fm != 0 && fm != 0xffu));
    for (uint32_t c = 0; c < 8; ++c) {
      if (!(cm & (1u << c))) continue;
      const uint32_t id = r[2 + c];
      ok = ok && id >= 2u && id - 2u < child_count;
      w[1 + k++] = ok ? child_refs[id - 2u] : kEmptyRef;
    }
    if (!ok) {
      set_status(&t.hdr->status, kDevInvalid);
      new_refs[i] = kEmptyRef;
      continue;
    }
    new_refs[i] = unique_insert_node(t, l, w, 1 + k, offsets[i]);
  }
}

__global__ void import_finish_kernel(Tables t, uint32_t l, uint32_t n, const uint32_t *rec,
                                     const uint32_t *offsets) {
  t.hdr->node_count[l] = n;
  if (l < t.depth)
    t.hdr->pool_used[l] = n ? offsets[n - 1] + 1u + __popc(rec[(n - 1) * 10ull] & 0xffu) : 0u;
}

__global__ void import_root_kernel(Tables t, const uint32_t *level0_refs, uint32_t root_id) {
  if (t.hdr->status != kDevOk) return;
  t.hdr->root = root_id >= 2u ? level0_refs[root_id - 2u] : root_id;
}

// The level's node count and pool use, once its items are in.
__global__ void finish_level_kernel(Tables t, uint32_t l, LevelMarks m, const uint32_t *staged,
                                    const uint32_t *offsets) {
  const uint32_t n = *m.live;
  t.hdr->node_count[l] = n;
  if (l < t.depth)
    t.hdr->pool_used[l] = n ? offsets[n - 1] + 1u + __popc(staged[(n - 1) * 9ull] & 0xffu) : 0u;
}

__global__ void seed_root_kernel(LevelMarks m, uint32_t root) {
  m.refs[0] = root;
  *m.live = 1;
}

__global__ void set_root_kernel(Tables t, uint32_t root) { t.hdr->root = root; }

__global__ void publish_compacted_root_kernel(Tables t, LevelMarks m0) {
  if (t.hdr->status == kDevOk) t.hdr->root = m0.new_refs[0];
}

// Carver stand-in that only adds up sizes (pointers come back null).
struct SizingCarver {
  Sizer z;
  template <class T> T *take(size_t n) {
    z.take<T>(n);
    return nullptr;
  }
};

// ------------------------------------------------------------ item set --
// A standalone content-addressed store of fixed-width items (the reference's
// AccelerationHashSet32, cuda/hash_table/acceleration_hash/set/*): one table
// of the same kind as a DAG level.  Pointers are item index + 1 (0 = null).

__device__ __forceinline__ uint32_t item_ptr(uint32_t ref, uint32_t width) {
  return ref >= 2u ? (ref - 2u) / width + 1u : 0u;
}

// Probe only: the ref of an equal item, or 0.
__device__ uint32_t node_find(const Tables &t, uint32_t l, const uint32_t *w, uint32_t n) {
  const uint64_t h = hash_words(w, n);
  const uint32_t tag = static_cast<uint32_t>(h >> 32) | 1u;
  const uint64_t *idx = t.index[l];
  const uint32_t *pool = t.pool[l];
  uint64_t pos = h & t.index_mask[l];
  for (uint32_t probe = 0; probe < kMaxProbes; ++probe) {
    const uint64_t v = ld_relaxed_u64(idx + pos);
    if (v == 0) return 0u;
    const uint32_t r = static_cast<uint32_t>(v);
    if (static_cast<uint32_t>(v >> 32) == tag && r >= 2u && r != kBusy) {
      fence_acq_rel_gpu();
      bool eq = true;
      for (uint32_t i = 0; i < n && eq; ++i) eq = pool[r - 2u + i] == w[i];
      if (eq) return r;
    }
    pos = (pos + 1) & t.index_mask[l];
  }
  return 0u;
}

enum class ItemOp { Find, FindOrInsert, InsertUnique };

template <ItemOp Op>
__global__ void itemset_kernel(Tables t, uint32_t width, const uint32_t *items, uint32_t n,
                               uint32_t *ptrs, uint32_t *statuses) {
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint32_t w[9];
    for (uint32_t j = 0; j < width; ++j) w[j] = items[i * width + j];
    uint32_t ref = 0, status = VX_HASH_NOT_FOUND;
    if (Op == ItemOp::Find) {
      ref = node_find(t, 0, w, width);
      status = ref ? VX_HASH_FOUND : VX_HASH_NOT_FOUND;
    } else if (Op == ItemOp::FindOrInsert) {
      bool inserted = false;
      ref = node_find_or_insert(t, 0, ArrayWords{w, width}, &inserted);
      status = ref >= 2u ? (inserted ? VX_HASH_INSERTED : VX_HASH_FOUND) : VX_HASH_OVERFLOW;
      if (ref < 2u) ref = 0;
    } else {
      const uint32_t off = atomicAdd(&t.hdr->pool_used[0], width);
      if (static_cast<uint64_t>(off) + width > t.pool_cap[0]) {
        status = VX_HASH_OVERFLOW;
      } else {
        ref = unique_insert_node(t, 0, w, width, off);
        status = VX_HASH_INSERTED;
        atomicAdd(reinterpret_cast<unsigned long long *>(&t.hdr->node_count[0]), 1ull);
      }
    }
    ptrs[i] = item_ptr(ref, width);
    if (statuses) statuses[i] = status;
  }
}

__global__ void itemset_read_kernel(Tables t, uint32_t width, const uint32_t *ptrs, uint32_t n,
                                    uint32_t *out, uint32_t *statuses) {
  const uint32_t stored = t.hdr->pool_used[0] / width;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint32_t p = ptrs[i];
    const bool ok = p >= 1u && p <= stored;
    for (uint32_t j = 0; j < width; ++j)
      out[i * width + j] = ok ? t.pool[0][(p - 1u) * static_cast<uint64_t>(width) + j] : 0u;
    if (statuses) statuses[i] = ok ? VX_HASH_FOUND : VX_HASH_NOT_FOUND;
  }
}

} // namespace vx::dag

struct vx_itemset {
  vx::dag::Tables t{};
  uint32_t width = 0;
  uint64_t index_slots = 0;
};

namespace {
template <vx::dag::ItemOp Op>
vx_status itemset_launch(const vx_itemset *s, const uint32_t *items, uint32_t count,
                         uint32_t *ptrs, uint32_t *statuses, vx_stream stream) {
  if (s == nullptr || ((items == nullptr || ptrs == nullptr) && count != 0))
    return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint32_t grid = std::min<uint32_t>(vx::ceil_div(count, vx::dag::kBlock),
                                           static_cast<uint32_t>(vx::sm_count()) * 16u);
  vx::prof::Scope sc("itemset", st);
  vx::dag::itemset_kernel<Op><<<grid, vx::dag::kBlock, 0, st>>>(s->t, s->width, items, count,
                                                                 ptrs, statuses);
  return vx::from_cuda(cudaGetLastError());
}
} // namespace

extern "C" {

vx_status vx_itemset_clear(vx_itemset *s, vx_stream stream) {
  if (s == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  VX_TRY_CUDA(cudaMemsetAsync(s->t.index[0], 0, s->index_slots * 8, st));
  VX_TRY_CUDA(cudaMemsetAsync(s->t.hdr, 0, sizeof(vx::edit::Header), st));
  return VX_OK;
}

vx_status vx_itemset_destroy(vx_itemset *s) {
  if (s == nullptr) return VX_ERR_INVALID_VALUE;
  cudaFree(s->t.index[0]);
  cudaFree(s->t.pool[0]);
  cudaFree(s->t.hdr);
  delete s;
  return VX_OK;
}

vx_status vx_itemset_create(uint32_t width, uint32_t max_items, vx_itemset **out) {
  if (out == nullptr || width < 1 || width > 9 || max_items == 0) return VX_ERR_INVALID_VALUE;
  auto *s = new (std::nothrow) vx_itemset;
  if (s == nullptr) return VX_ERR_MEMORY_ALLOCATION;
  s->width = width;
  s->t.depth = 1;
  s->index_slots = vx::dag::next_pow2(2ull * max_items);
  s->t.index_mask[0] = s->index_slots - 1;
  s->t.pool_cap[0] = std::min<uint64_t>(static_cast<uint64_t>(max_items) * width, 0xfffffff0ull);
  cudaError_t e = cudaMalloc(&s->t.index[0], s->index_slots * 8);
  if (e == cudaSuccess) e = cudaMalloc(&s->t.pool[0], s->t.pool_cap[0] * 4);
  if (e == cudaSuccess) e = cudaMalloc(&s->t.hdr, sizeof(vx::edit::Header));
  if (e != cudaSuccess) {
    vx_itemset_destroy(s);
    return vx::from_cuda(e);
  }
  const vx_status st = vx_itemset_clear(s, nullptr);
  if (st != VX_OK) {
    vx_itemset_destroy(s);
    return st;
  }
  VX_TRY_CUDA(cudaStreamSynchronize(nullptr));
  *out = s;
  return VX_OK;
}


vx_status vx_itemset_find(const vx_itemset *s, const uint32_t *items, uint32_t count,
                          uint32_t *ptrs, uint32_t *statuses, vx_stream stream) {
  return itemset_launch<vx::dag::ItemOp::Find>(s, items, count, ptrs, statuses, stream);
}

vx_status vx_itemset_find_or_insert(vx_itemset *s, const uint32_t *items, uint32_t count,
                                    uint32_t *ptrs, uint32_t *statuses, vx_stream stream) {
  return itemset_launch<vx::dag::ItemOp::FindOrInsert>(s, items, count, ptrs, statuses, stream);
}

vx_status vx_itemset_insert_unique_unchecked(vx_itemset *s, const uint32_t *items,
                                             uint32_t count, uint32_t *ptrs,
                                             uint32_t *statuses, vx_stream stream) {
  return itemset_launch<vx::dag::ItemOp::InsertUnique>(s, items, count, ptrs, statuses, stream);
}

vx_status vx_itemset_read(const vx_itemset *s, const uint32_t *ptrs, uint32_t count,
                          uint32_t *items, uint32_t *statuses, vx_stream stream) {
  if (s == nullptr || ((items == nullptr || ptrs == nullptr) && count != 0))
    return VX_ERR_INVALID_VALUE;
  if (count == 0) return VX_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uint32_t grid = std::min<uint32_t>(vx::ceil_div(count, vx::dag::kBlock),
                                           static_cast<uint32_t>(vx::sm_count()) * 16u);
  vx::prof::Scope sc("itemset_read", st);
  vx::dag::itemset_read_kernel<<<grid, vx::dag::kBlock, 0, st>>>(s->t, s->width, ptrs, count,
                                                                 items, statuses);
  return vx::from_cuda(cudaGetLastError());
}

vx_status vx_itemset_count(const vx_itemset *s, uint64_t *host_count, vx_stream stream) {
  if (s == nullptr || host_count == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  VX_TRY_CUDA(cudaMemcpyAsync(host_count, &s->t.hdr->node_count[0], 8, cudaMemcpyDeviceToHost, st));
  VX_TRY_CUDA(cudaStreamSynchronize(st));
  return VX_OK;
}

vx_status vx_dag_import_canonical(vx_dag *d, uint32_t root, const uint64_t *host_counts,
                                  const uint32_t *host_nodes, const uint64_t *host_leaves,
                                  vx_stream stream) {
  if (d == nullptr || host_counts == nullptr || root > 2u) return VX_ERR_INVALID_VALUE;
  const uint32_t D = d->t.depth;
  uint64_t total_nodes = 0, max_n = 1;
  for (uint32_t l = 0; l <= D; ++l) {
    if (host_counts[l] > 0xffffffffull) return VX_ERR_CAPACITY;
    if (l < D) total_nodes += host_counts[l];
    max_n = std::max<uint64_t>(max_n, host_counts[l]);
  }
  if ((total_nodes && host_nodes == nullptr) || (host_counts[D] && host_leaves == nullptr))
    return VX_ERR_INVALID_VALUE;
  if (root == 2u && host_counts[0] != 1) return VX_ERR_INVALID_VALUE;
  if (root < 2u && total_nodes + host_counts[D] != 0) return VX_ERR_INVALID_VALUE;
  uint64_t rec0 = 0;
  for (uint32_t l = 0; l < D; ++l) {
    uint64_t words = 0; // exact pool words of the level
    for (uint64_t i = 0; i < host_counts[l]; ++i)
      words += 1 + __builtin_popcount(host_nodes[(rec0 + i) * 10] & 0xffu);
    rec0 += host_counts[l];
    if (host_counts[l] > d->index_slots[l] / 2 || words > d->t.pool_cap[l])
      return VX_ERR_CAPACITY;
  }
  if (host_counts[D] > d->leaf_slots / 2) return VX_ERR_CAPACITY;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t grid = static_cast<uint32_t>(vx::sm_count()) * 8u;
  // One temporary block: records of the largest level, its offsets, new
  // refs of two adjacent levels, the leaf masks and the scan workspace.
  const size_t scan_bytes = vx_scan_workspace_size(static_cast<uint32_t>(max_n));
  vx::Sizer z;
  z.take<uint32_t>(max_n * 10);
  z.take<uint32_t>(max_n);
  z.take<uint32_t>(max_n);
  z.take<uint32_t>(max_n);
  z.take<uint64_t>(std::max<uint64_t>(host_counts[D], 1));
  z.take<unsigned char>(scan_bytes);
  struct TempBlock {
    void *p = nullptr;
    ~TempBlock() { if (p) cudaFree(p); }
  } temp;
  VX_TRY_CUDA(cudaMalloc(&temp.p, z.offset));
  vx::Carver c(temp.p);
  uint32_t *rec = c.take<uint32_t>(max_n * 10);
  uint32_t *offsets = c.take<uint32_t>(max_n);
  uint32_t *refs[2] = {c.take<uint32_t>(max_n), c.take<uint32_t>(max_n)};
  uint64_t *masks = c.take<uint64_t>(std::max<uint64_t>(host_counts[D], 1));
  void *scan_ws = c.take<unsigned char>(scan_bytes);
  VX_TRY(vx_dag_reset(d, stream));
  const uint32_t nl = static_cast<uint32_t>(host_counts[D]);
  if (nl) {
    VX_TRY_CUDA(cudaMemcpyAsync(masks, host_leaves, nl * 8ull, cudaMemcpyHostToDevice, s));
    vx::prof::Scope sc("dag_import", s);
    import_leaves_kernel<<<grid, kBlock, 0, s>>>(d->t, masks, nl, refs[D & 1u]);
    VX_TRY_CUDA(cudaGetLastError());
  }
  import_finish_kernel<<<1, 1, 0, s>>>(d->t, D, nl, nullptr, nullptr);
  VX_TRY_CUDA(cudaGetLastError());
  std::vector<uint64_t> first(D + 1, 0); // first record of each level
  for (uint32_t l = 1; l < D; ++l) first[l] = first[l - 1] + host_counts[l - 1] * 10;
  for (uint32_t r = D; r > 0; --r) {
    const uint32_t l = r - 1;
    const uint32_t n = static_cast<uint32_t>(host_counts[l]);
    if (n) {
      VX_TRY_CUDA(cudaMemcpyAsync(rec, host_nodes + first[l], n * 40ull, cudaMemcpyHostToDevice,
                                  s));
      {
        vx::prof::Scope sc("dag_import", s);
        import_words_kernel<<<grid, kBlock, 0, s>>>(rec, n, offsets);
        VX_TRY_CUDA(cudaGetLastError());
      }
      VX_TRY(vx_scan_exclusive_sum_u32(offsets, n, scan_ws, scan_bytes, s));
      vx::prof::Scope sc("dag_import", s);
      import_nodes_kernel<<<grid, kBlock, 0, s>>>(d->t, l, rec, n, refs[(l + 1) & 1u],
                                                  static_cast<uint32_t>(host_counts[l + 1]),
                                                  offsets, refs[l & 1u]);
      VX_TRY_CUDA(cudaGetLastError());
    }
    import_finish_kernel<<<1, 1, 0, s>>>(d->t, l, n, rec, offsets);
    VX_TRY_CUDA(cudaGetLastError());
  }
  import_root_kernel<<<1, 1, 0, s>>>(d->t, refs[0], root);
  VX_TRY_CUDA(cudaGetLastError());
  return read_status(d, s, true);
}

namespace {
constexpr char kDagFileMagic[8] = {'V', 'X', 'D', 'A', 'G', 'C', 'N', '1'};
} // namespace

vx_status vx_dag_save(const vx_dag *d, const char *path, vx_stream stream) {
  if (d == nullptr || path == nullptr) return VX_ERR_INVALID_VALUE;
  const uint32_t D = d->t.depth;
  uint32_t root = 0;
  std::vector<uint64_t> counts(D + 1, 0);
  VX_TRY(vx_dag_export_canonical(d, &root, counts.data(), nullptr, 0, nullptr, 0, stream));
  uint64_t words = 0;
  for (uint32_t l = 0; l < D; ++l) words += counts[l] * 10;
  std::vector<uint32_t> nodes(words);
  std::vector<uint64_t> leaves(counts[D]);
  VX_TRY(vx_dag_export_canonical(d, &root, counts.data(), nodes.data(), words, leaves.data(),
                                 leaves.size(), stream));
  FILE *f = std::fopen(path, "wb");
  if (f == nullptr) return VX_ERR_IO;
  const uint32_t head[4] = {1u /* version */, D, root, 0u};
  bool ok = std::fwrite(kDagFileMagic, 1, 8, f) == 8 && std::fwrite(head, 4, 4, f) == 4 &&
            std::fwrite(counts.data(), 8, counts.size(), f) == counts.size() &&
            std::fwrite(nodes.data(), 4, nodes.size(), f) == nodes.size() &&
            std::fwrite(leaves.data(), 8, leaves.size(), f) == leaves.size();
  ok = std::fclose(f) == 0 && ok;
  return ok ? VX_OK : VX_ERR_IO;
}

vx_status vx_dag_load(vx_dag *d, const char *path, vx_stream stream) {
  if (d == nullptr || path == nullptr) return VX_ERR_INVALID_VALUE;
  FILE *f = std::fopen(path, "rb");
  if (f == nullptr) return VX_ERR_IO;
  struct Closer {
    FILE *f;
    ~Closer() { std::fclose(f); }
  } closer{f};
  char magic[8];
  uint32_t head[4];
  if (std::fread(magic, 1, 8, f) != 8 || std::memcmp(magic, kDagFileMagic, 8) != 0 ||
      std::fread(head, 4, 4, f) != 4 || head[0] != 1u)
    return VX_ERR_INVALID_VALUE;
  const uint32_t D = head[1], root = head[2];
  if (D != d->t.depth || root > 2u) return VX_ERR_INVALID_VALUE;
  std::vector<uint64_t> counts(D + 1);
  if (std::fread(counts.data(), 8, counts.size(), f) != counts.size()) return VX_ERR_IO;
  uint64_t words = 0;
  for (uint32_t l = 0; l < D; ++l) {
    if (counts[l] > (1ull << 32)) return VX_ERR_INVALID_VALUE;
    words += counts[l] * 10;
  }
  if (counts[D] > (1ull << 32)) return VX_ERR_INVALID_VALUE;
  std::vector<uint32_t> nodes(words);
  std::vector<uint64_t> leaves(counts[D]);
  if (std::fread(nodes.data(), 4, nodes.size(), f) != nodes.size() ||
      std::fread(leaves.data(), 8, leaves.size(), f) != leaves.size())
    return VX_ERR_IO;
  return vx_dag_import_canonical(d, root, counts.data(), nodes.data(), leaves.data(), stream);
}

vx_status vx_dag_compact(vx_dag *d, vx_stream stream) {
  if (d == nullptr) return VX_ERR_INVALID_VALUE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t D = d->t.depth;
  vx::edit::Header h;
  VX_TRY_CUDA(cudaMemcpyAsync(&h, d->t.hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  if (h.status != vx::kDevOk) return vx::status_from_device(h.status);
  if (h.root < 2) { // empty or full world: nothing is live
    VX_TRY(vx_dag_reset(d, stream));
    vx::prof::Scope sc("dag_set_root", s);
    set_root_kernel<<<1, 1, 0, s>>>(d->t, h.root);
    return vx::from_cuda(cudaGetLastError());
  }
  const uint32_t grid = static_cast<uint32_t>(vx::sm_count()) * 8u;
  // Temporaries: per level a bitmap and prefix over its old ref space and
  // live-ref / new-ref lists sized by the level's node count, the scan
  // workspace, then (once the live counts are known) the staged items.  They
  // live in the idle edit arena when it is large enough, else in temporary
  // allocations.
  std::vector<LevelMarks> m(D + 1);
  uint64_t max_words = 1;
  for (uint32_t l = 0; l <= D; ++l) {
    const uint64_t space = l == D ? d->leaf_slots
                                  : std::min<uint64_t>(h.pool_used[l], d->t.pool_cap[l]);
    m[l].words = std::max<uint64_t>((space + 31) / 32, 1);
    m[l].cap = static_cast<uint32_t>(std::max<uint64_t>(h.node_count[l], 1));
    max_words = std::max(max_words, m[l].words);
  }
  if (max_words > 0xffffffffull) return VX_ERR_CAPACITY;
  uint64_t max_scan = max_words;
  for (uint32_t l = 0; l <= D; ++l) max_scan = std::max<uint64_t>(max_scan, m[l].cap);
  const size_t scan_bytes = vx_scan_workspace_size(static_cast<uint32_t>(max_scan));
  uint32_t *counts = nullptr;
  void *scan_ws = nullptr;
  auto carve_marks = [&](auto &c) {
    counts = c.template take<uint32_t>(D + 1);
    scan_ws = c.template take<unsigned char>(scan_bytes);
    for (uint32_t l = 0; l <= D; ++l) {
      m[l].live = counts + l;
      m[l].bits = c.template take<uint32_t>(2 * m[l].words);
      m[l].prefix = c.template take<uint32_t>(m[l].words);
      m[l].refs = c.template take<uint32_t>(m[l].cap);
      m[l].new_refs = c.template take<uint32_t>(m[l].cap);
    }
  };
  const size_t arena_bytes = static_cast<size_t>(d->a.item_cap) * sizeof(vx::edit::Item) +
                             2ull * d->a.pair_cap * 4;
  struct TempBlock {
    void *p = nullptr;
    ~TempBlock() { if (p) cudaFree(p); }
  } temp_marks, temp_staged;
  SizingCarver marks_size;
  carve_marks(marks_size);
  void *marks_base = d->arena_mem;
  if (marks_size.z.offset > arena_bytes) {
    VX_TRY_CUDA(cudaMalloc(&temp_marks.p, marks_size.z.offset));
    marks_base = temp_marks.p;
  }
  vx::Carver carver(marks_base);
  carve_marks(carver);
  for (uint32_t l = 1; l <= D; ++l)
    VX_TRY_CUDA(cudaMemsetAsync(m[l].bits, 0, m[l].words * 8, s));
  {
    vx::prof::Scope sc("dag_compact_mark", s);
    seed_root_kernel<<<1, 1, 0, s>>>(m[0], h.root);
  }
  VX_TRY_CUDA(cudaGetLastError());
  // Mark top-down: children of level l's live items, then rank level l+1.
  for (uint32_t l = 0; l < D; ++l) {
    {
      vx::prof::Scope sc("dag_compact_mark", s);
      mark_children_kernel<<<grid, kBlock, 0, s>>>(d->t, l, m[l], m[l + 1]);
      VX_TRY_CUDA(cudaGetLastError());
    }
    {
      vx::prof::Scope sc("dag_compact_rank", s);
      popcount_kernel<<<grid, kBlock, 0, s>>>(m[l + 1]);
      VX_TRY_CUDA(cudaGetLastError());
    }
    VX_TRY(vx_scan_exclusive_sum_u32(m[l + 1].prefix, static_cast<uint32_t>(m[l + 1].words),
                                     scan_ws, scan_bytes, s));
    {
      vx::prof::Scope sc("dag_compact_rank", s);
      list_kernel<<<grid, kBlock, 0, s>>>(d->t, m[l + 1]);
      VX_TRY_CUDA(cudaGetLastError());
    }
  }
  // Live counts (and a capacity error raised while listing, which must not
  // be lost to the reset below).
  std::vector<uint32_t> live(D + 1, 0);
  uint32_t mark_status = 0;
  VX_TRY_CUDA(cudaMemcpyAsync(live.data(), counts, 4 * (D + 1), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaMemcpyAsync(&mark_status, &d->t.hdr->status, 4, cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  if (mark_status != vx::kDevOk) return vx::status_from_device(mark_status);
  // Staging, sized by the live counts: 9 words per inner item, leaf masks.
  std::vector<uint32_t *> staged(D + 1, nullptr), offsets(D + 1, nullptr);
  uint64_t *leaf_masks = nullptr;
  auto carve_staged = [&](auto &c) {
    leaf_masks = c.template take<uint64_t>(std::max<uint32_t>(live[D], 1));
    for (uint32_t l = 0; l < D; ++l) {
      staged[l] = c.template take<uint32_t>(std::max<uint32_t>(live[l], 1) * 9ull);
      offsets[l] = c.template take<uint32_t>(std::max<uint32_t>(live[l], 1));
    }
  };
  SizingCarver staged_size;
  staged_size.z.offset = marks_base == d->arena_mem ? carver.offset : 0;
  carve_staged(staged_size);
  if (marks_base == d->arena_mem && staged_size.z.offset <= arena_bytes) {
    carve_staged(carver);
  } else {
    SizingCarver alone;
    carve_staged(alone);
    VX_TRY_CUDA(cudaMalloc(&temp_staged.p, alone.z.offset));
    vx::Carver c2(temp_staged.p);
    carve_staged(c2);
  }
  // Stage every live item, then clear the tables.
  for (uint32_t l = 0; l <= D; ++l) {
    vx::prof::Scope sc("dag_compact_stage", s);
    stage_kernel<<<grid, kBlock, 0, s>>>(d->t, l, m[l], staged[l], leaf_masks);
    VX_TRY_CUDA(cudaGetLastError());
  }
  VX_TRY(vx_dag_reset(d, stream));
  // Re-insert bottom-up; a child's new ref is new_refs[rank(old ref)].
  for (uint32_t r = D + 1; r > 0; --r) {
    const uint32_t l = r - 1;
    if (l < D && live[l]) {
      {
        vx::prof::Scope sc("dag_compact_reinsert", s);
        item_words_kernel<<<grid, kBlock, 0, s>>>(m[l], staged[l], offsets[l]);
        VX_TRY_CUDA(cudaGetLastError());
      }
      VX_TRY(vx_scan_exclusive_sum_u32(offsets[l], live[l], scan_ws, scan_bytes, s));
    }
    vx::prof::Scope sc("dag_compact_reinsert", s);
    if (l == D)
      reinsert_leaves_kernel<<<grid, kBlock, 0, s>>>(d->t, m[D], leaf_masks);
    else
      reinsert_nodes_kernel<<<grid, kBlock, 0, s>>>(d->t, l, m[l], m[l + 1], staged[l],
                                                    offsets[l]);
    VX_TRY_CUDA(cudaGetLastError());
    finish_level_kernel<<<1, 1, 0, s>>>(d->t, l, m[l], staged[l], offsets[l]);
    VX_TRY_CUDA(cudaGetLastError());
  }
  {
    vx::prof::Scope sc("dag_set_root", s);
    publish_compacted_root_kernel<<<1, 1, 0, s>>>(d->t, m[0]);
  }
  VX_TRY_CUDA(cudaGetLastError());
  return read_status(d, s, true);
}

} // extern "C"

// ======================================================= serving hooks ==

#include "dag_internal.cuh"

namespace vx::dag {

const void *device_header(const vx_dag *d) { return d->t.hdr; }
size_t header_bytes() { return sizeof(vx::edit::Header); }
uint32_t header_root(const void *hh) { return static_cast<const vx::edit::Header *>(hh)->root; }
uint32_t header_status(const void *hh) { return static_cast<const vx::edit::Header *>(hh)->status; }

TableRoom table_room(const vx_dag *d, const void *hh) {
  const auto *h = static_cast<const vx::edit::Header *>(hh);
  TableRoom r{};
  r.depth = d->t.depth;
  for (uint32_t l = 0; l < d->t.depth; ++l) {
    r.node_cap[l] = d->index_slots[l] / 2;
    r.word_cap[l] = d->t.pool_cap[l];
    r.nodes[l] = h->node_count[l];
    r.words[l] = h->pool_used[l];
  }
  r.node_cap[d->t.depth] = d->leaf_slots / 2;
  r.nodes[d->t.depth] = h->node_count[d->t.depth];
  return r;
}

vx_status read_header(const vx_dag *d, void *host, cudaStream_t s) {
  VX_TRY_CUDA(cudaMemcpyAsync(host, d->t.hdr, sizeof(vx::edit::Header), cudaMemcpyDeviceToHost, s));
  VX_TRY_CUDA(cudaStreamSynchronize(s));
  return VX_OK;
}

double fill_fraction(const vx_dag *d, const void *hh) {
  const auto *h = static_cast<const vx::edit::Header *>(hh);
  double f = 0.0;
  for (uint32_t l = 0; l < d->t.depth; ++l) {
    f = std::max(f, static_cast<double>(h->node_count[l]) / (d->index_slots[l] / 2.0));
    f = std::max(f, static_cast<double>(h->pool_used[l]) / static_cast<double>(d->t.pool_cap[l]));
  }
  f = std::max(f, static_cast<double>(h->node_count[d->t.depth]) / (d->leaf_slots / 2.0));
  return f;
}

} // namespace vx::dag
