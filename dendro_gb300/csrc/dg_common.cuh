// Shared device/host helpers for the GB300 octree hot path.
//
// Octant keys: the Morton (bit-interleaved, z above y above x) index of the
// anchor at the finest level D, right-aligned in a 128-bit value; an octant
// at level l has its low 3*(D-l) key bits zero.  Linear octrees are stored as
// a key array plus a level array (one byte per octant); since a linear
// octree never holds two octants with the same anchor, the key alone orders
// it exactly like the reference's TreeNode::operator< (TreeNode.tcc:211-236).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstddef>

#include "dendro_gb300.h"

namespace dg {

typedef unsigned __int128 u128;

struct __align__(16) Key128 {
  uint64_t lo, hi;
};

__host__ __device__ __forceinline__ u128 to_u128(Key128 k) { return ((u128)k.hi << 64) | (u128)k.lo; }
__host__ __device__ __forceinline__ Key128 from_u128(u128 v) {
  Key128 k;
  k.lo = (uint64_t)v;
  k.hi = (uint64_t)(v >> 64);
  return k;
}
__host__ __device__ __forceinline__ bool key_eq(Key128 a, Key128 b) { return a.lo == b.lo && a.hi == b.hi; }
__host__ __device__ __forceinline__ bool key_lt(Key128 a, Key128 b) {
  return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo);
}
__host__ __device__ __forceinline__ bool key_le(Key128 a, Key128 b) { return !key_lt(b, a); }

// Bit i of a coordinate is bit 3 i of its axis in the key.  In pieces of 10
// bits, 30 of the key: 32-bit steps, of which the GPU does half as many as of
// 64-bit ones on pieces of 21 (records of 8.8e7 octants 0.67 -> 0.57 ms).
// spread the low 10 bits of v to every third bit
__host__ __device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | v << 16) & 0x030000ffu;
  v = (v | v << 8) & 0x0300f00fu;
  v = (v | v << 4) & 0x030c30c3u;
  return (v | v << 2) & 0x09249249u;
}
// inverse of spread10
__host__ __device__ __forceinline__ uint32_t compact10(uint32_t v) {
  v &= 0x09249249u;
  v = (v | v >> 2) & 0x030c30c3u;
  v = (v | v >> 4) & 0x0300f00fu;
  v = (v | v >> 8) & 0x030000ffu;
  return (v | v >> 16) & 0x3ffu;
}

// Morton key of 32-bit coordinates (96 bits used)
__host__ __device__ __forceinline__ Key128 morton3(uint32_t x, uint32_t y, uint32_t z) {
  uint32_t p[3];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int i = 0; i < 3; i++)
    p[i] = spread10(x >> 10 * i) | spread10(y >> 10 * i) << 1 | spread10(z >> 10 * i) << 2;
  const uint32_t t = (x >> 30 & 1u) | (y >> 30 & 1u) << 1 | (z >> 30 & 1u) << 2 | (x >> 31) << 3 | (y >> 31) << 4 |
                     (z >> 31) << 5;  // coordinate bits 30 and 31
  Key128 k;
  k.lo = (uint64_t)p[0] | (uint64_t)p[1] << 30 | (uint64_t)p[2] << 60;
  k.hi = (uint64_t)p[2] >> 4 | (uint64_t)t << 26;
  return k;
}

__host__ __device__ __forceinline__ void demorton3(Key128 k, uint32_t &x, uint32_t &y, uint32_t &z) {
  const uint32_t p[3] = {(uint32_t)k.lo, (uint32_t)(k.lo >> 30), (uint32_t)(k.lo >> 60) | (uint32_t)k.hi << 4};
  const uint32_t t = (uint32_t)(k.hi >> 26);
  x = (t & 1u) << 30 | (t >> 3 & 1u) << 31;
  y = (t >> 1 & 1u) << 30 | (t >> 4 & 1u) << 31;
  z = (t >> 2 & 1u) << 30 | (t >> 5 & 1u) << 31;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int i = 0; i < 3; i++) {
    x |= compact10(p[i]) << 10 * i;
    y |= compact10(p[i] >> 1) << 10 * i;
    z |= compact10(p[i] >> 2) << 10 * i;
  }
}

__host__ __device__ __forceinline__ Key128 key_shr(Key128 k, unsigned s) {
  if (s == 0) return k;
  if (s >= 128) return Key128{0, 0};
  if (s >= 64) return Key128{k.hi >> (s - 64), 0};
  return Key128{(k.lo >> s) | (k.hi << (64 - s)), k.hi >> s};
}
__host__ __device__ __forceinline__ Key128 key_shl(Key128 k, unsigned s) {
  if (s == 0) return k;
  if (s >= 128) return Key128{0, 0};
  if (s >= 64) return Key128{0, k.lo << (s - 64)};
  return Key128{k.lo << s, (k.hi << s) | (k.lo >> (64 - s))};
}
__host__ __device__ __forceinline__ Key128 key_or(Key128 a, Key128 b) { return Key128{a.lo | b.lo, a.hi | b.hi}; }
__host__ __device__ __forceinline__ Key128 key_xor(Key128 a, Key128 b) { return Key128{a.lo ^ b.lo, a.hi ^ b.hi}; }

// number of leading zero bits of k within a `bits`-wide field (bits <= 128)
__device__ __forceinline__ int key_clz(Key128 k, int bits) {
  int lz;
  if (k.hi) lz = __clzll((long long)k.hi);
  else if (k.lo) lz = 64 + __clzll((long long)k.lo);
  else lz = 128;
  return lz - (128 - bits);
}

// status codes: DG_OK / DG_ERR_* of the C ABI (include/dendro_gb300.h)

// device-side error flags (bitmask written by kernels, read by the host)
enum {
  DGF_DOMAIN = 1u,         // a point outside [0, gLen)^3 or not finite
  DGF_NOT_BALANCED = 2u,   // DA input not 2:1 balanced / not complete
  DGF_TIMEOUT = 4u,        // a bounded spin gave up
  DGF_INTERNAL = 8u,       // internal consistency check failed
  DGF_ORDER = 16u,         // input not sorted / unique as the caller declared
  DGF_LONG_RUN = 32u,      // a run of keys with one sorted prefix is too long to order in place
  DGF_CAPACITY = 64u,      // a table sized by estimate is full (the host retries with a larger one)
};

}  // namespace dg
