// Internal octants ("nodes") as sortable keys, and hash tables of them:
// shared by construction and balance (dg_octree.cu) and the mesh build
// (dg_da.cu).
#pragma once

#include "dg_octree.cuh"

namespace dg {

__device__ __forceinline__ void set_flag(uint32_t *flags, uint32_t f) { atomicOr(flags, f); }

// key with only the Morton bits of one cloud (bits [0, 3D))
__host__ __device__ __forceinline__ Key128 morton_part(Key128 k, unsigned D) {
  Key128 a = tag_anchor(k);
  if (3 * D < 64) {
    a.lo &= (3 * D) ? ((1ull << (3 * D)) - 1) : 0ull;
    a.hi = 0;
  } else {
    a.hi &= (1ull << (3 * D - 64)) - 1;
  }
  return a;
}
__host__ __device__ __forceinline__ uint64_t seg_of(Key128 k, unsigned D) {
  return to_u128(tag_anchor(k)) >> (3 * D) & 0xffffffffffull;
}
__host__ __device__ __forceinline__ Key128 seg_key(uint64_t seg, unsigned D) {
  return from_u128((u128)seg << (3 * D));
}

// NCA level of two points of the same cloud; -1 across clouds
__device__ __forceinline__ int nca_level(Key128 a, Key128 b, unsigned D) {
  Key128 x = key_xor(tag_anchor(a), tag_anchor(b));
  if (!x.lo && !x.hi) return (int)D;
  int lz = key_clz(x, 3 * (int)D);
  return lz < 0 ? -1 : lz / 3;
}

// A node: an internal octant of level <= Lm as one sortable key, its path (3
// bits per level to level Lm, the cloud index above) over 5 bits of level:
// preorder is key order.  64-bit keys where they suffice, else 128-bit.
__device__ __forceinline__ uint64_t node_wide(uint64_t k) { return k; }
__device__ __forceinline__ u128 node_wide(Key128 k) { return to_u128(k); }
// no node: the level bits of a node never are 31
__device__ __forceinline__ uint64_t node_empty(uint64_t) { return ~0ull; }
__device__ __forceinline__ u128 node_empty(u128) { return ~(u128)0; }
template <typename K>
struct NodeWide;
template <>
struct NodeWide<uint64_t> {
  typedef uint64_t W;
  __host__ __device__ __forceinline__ static uint64_t narrow(W w) { return w; }
  __device__ __forceinline__ static W of(Key128 k) { return k.lo; }
  __device__ __forceinline__ static Key128 key(W w) { return Key128{w, 0}; }
};
template <>
struct NodeWide<Key128> {
  typedef u128 W;
  __host__ __device__ __forceinline__ static Key128 narrow(W w) { return from_u128(w); }
  __device__ __forceinline__ static W of(Key128 k) { return to_u128(k); }
  __device__ __forceinline__ static Key128 key(W w) { return from_u128(w); }
};

// the ancestor of level l (<= Lm) of a tagged anchor at depth D
template <typename K>
__device__ __forceinline__ K node_of(Key128 anchor, unsigned l, unsigned Lm, unsigned D) {
  typedef NodeWide<K> N;
  const typename N::W idx = N::of(key_shr(anchor, 3 * (D - l)));
  return N::narrow(idx << (3 * (Lm - l)) << 5 | (typename N::W)l);
}

// Whether `next` may stand behind `prev` in the preorder list of an octree's
// nodes (or, with none, at its head): later, and a child of `prev` or of an
// ancestor of it, or the root of another cloud.  A list of which this holds all
// along has no node twice and every node's parent.
template <typename W>
__host__ __device__ __forceinline__ bool node_follows(bool any, W prev, W next, unsigned Lm) {
  const unsigned d = (unsigned)next & 31u;
  if (d > Lm || (any && next <= prev)) return false;
  if (d == 0) return ((next >> 5) & (((W)1 << (3 * Lm)) - 1)) == 0;
  const unsigned sh = 5 + 3 * (Lm - d + 1);  // to the parent's path
  return any && ((unsigned)prev & 31u) + 1 >= d && prev >> sh == next >> sh;
}

// sum of the octal digits of v
__device__ __forceinline__ unsigned digit_sum(uint64_t v) {
  const uint64_t m = 0x1249249249249249ull;  // bits 0, 3, ..., 60
  return __popcll(v & m) + 2 * __popcll(v & m << 1) + 4 * __popcll(v & m << 2) + (unsigned)(v >> 63);
}
__device__ __forceinline__ unsigned digit_sum(u128 v) {
  return digit_sum((uint64_t)((uint64_t)v & 0x7fffffffffffffffull)) + digit_sum((uint64_t)(v >> 63));
}

// whether node keys of octrees with leaves to level top (> 0) fit 64 bits
inline bool nodes_fit_64(unsigned top, unsigned seg_bits) { return 3 * (top - 1) + seg_bits + 5 <= 64; }

__device__ __forceinline__ uint64_t shfl_wide(uint64_t v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ u128 shfl_wide(u128 v, int lane) {
  return (u128)__shfl_sync(0xffffffffu, (uint64_t)(v >> 64), lane) << 64 | __shfl_sync(0xffffffffu, (uint64_t)v, lane);
}

// ---- the set of all nodes: open addressing.  The eight children of one
// octant share a group of eight slots (one cache line of 64-bit keys), as the
// candidates around one octant do; a probe goes to the next group's next slot,
// so that it leaves its child number's slots: on a face of the domain only four
// child numbers occur, on an edge two (stepping by 8, 981 of the 2,005 nodes of
// 1,000 points on an edge found no slot in a table of 4,096; stepping by 9 the
// longest search takes 10 steps, and at most 32 in 5.2e5 slots for 2.5e5 nodes of
// points on a face).  A bounded number of probes (NODE_PROBES; then DGF_CAPACITY,
// and the host retries with a larger table).
constexpr int NODE_PROBES = 512;
constexpr uint64_t NODE_STEP = 9;  // odd: all slots are reached

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 32;
  x *= 0xd6e8feb86659fd93ull;
  x ^= x >> 32;
  return x;
}
__device__ __forceinline__ uint64_t node_hash(uint64_t k, unsigned Lm) {
  const unsigned l = (unsigned)k & 31u, sh = 5 + 3 * (Lm - l);
  return mix64((k >> sh >> 3) * 32 + l) << 3 | (k >> sh & 7u);
}
__device__ __forceinline__ uint64_t node_hash(u128 k, unsigned Lm) {
  const unsigned l = (unsigned)k & 31u, sh = 5 + 3 * (Lm - l);
  const u128 par = k >> sh >> 3;
  return mix64(((uint64_t)par ^ (uint64_t)(par >> 64) * 0x9e3779b97f4a7c15ull) * 32 + l) << 3 | ((uint64_t)(k >> sh) & 7u);
}
// compare-and-swap of one slot, returning what it held
__device__ __forceinline__ uint64_t slot_cas(uint64_t *slot, uint64_t key) {
  const uint64_t cur = __ldcg(slot);  // a full slot never changes
  if (cur != ~0ull) return cur;
  return atomicCAS(reinterpret_cast<unsigned long long *>(slot), ~0ull, (unsigned long long)key);
}
__device__ __forceinline__ u128 slot_cas(Key128 *slot, u128 key) {
  uint64_t lo, hi;
  asm volatile("{\n\t.reg .b128 d, b, c;\n\t"
               "mov.b128 b, {%3, %4};\n\tmov.b128 c, {%5, %6};\n\t"
               "atom.relaxed.gpu.cas.b128 d, [%2], b, c;\n\tmov.b128 {%0, %1}, d;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(slot), "l"(~0ull), "l"(~0ull), "l"((uint64_t)key), "l"((uint64_t)(key >> 64))
               : "memory");
  return (u128)hi << 64 | lo;
}

// true when this call put the key into the table
template <typename K>
__device__ __forceinline__ bool node_insert(K *__restrict__ tab, uint64_t mask, typename NodeWide<K>::W key,
                                            unsigned Lm, uint32_t *flags) {
  uint64_t h = node_hash(key, Lm) & mask;
  for (int probe = 0; probe < NODE_PROBES; probe++) {
    const auto cur = slot_cas(tab + h, key);
    if (cur == node_empty(key)) return true;
    if (cur == key) return false;
    h = (h + NODE_STEP) & mask;
  }
  set_flag(flags, DGF_CAPACITY);
  return false;
}

// index of a key in a table filled by k_node_table, or NODE_NONE
constexpr uint32_t NODE_NONE = 0xffffffffu;
template <typename K>
__device__ __forceinline__ uint32_t node_find(const K *__restrict__ tab, const uint32_t *__restrict__ val,
                                              uint64_t mask, typename NodeWide<K>::W key, unsigned Lm) {
  uint64_t h = node_hash(key, Lm) & mask;
  for (int probe = 0; probe < NODE_PROBES; probe++) {
    const auto cur = node_wide(tab[h]);
    if (cur == key) return val[h];
    if (cur == node_empty(key)) return NODE_NONE;
    h = (h + NODE_STEP) & mask;
  }
  return NODE_NONE;
}

}  // namespace dg
