// Octree construction (points2Octree) and 2:1 balance (balanceOctree) on
// the GPU.  All data stays in HBM; the host only reads sizes.
//
// Batches: several clouds ("segments") are processed by the same launches;
// segment s lives in key bits [3D, 3D + seg_bits) (dg_octree.cuh), so every
// sort, NCA and gap computation below stays inside its own cloud.
//
// Both pipelines describe an octree by its internal octants ("nodes"), sorted
// in preorder, and write the leaves from them (k_emit_leaves): with i the
// preorder index of a node of level d and digits(.) the sum of its path's
// child numbers, 7 (i - d) + digits leaves precede it, so every leaf's place
// follows from the nodes before it and no leaf is sorted or counted.
//
// Construction (unique points, reference p2oLocal, src/construct.cpp:976):
// the leaf that holds point i is the child of its deepest ancestor that
// contains more than maxPts points.  With the points in Morton order that
// ancestor's level is max_j NCA(p_j, p_{j+m}) over the windows j in
// [i-m, i] (m = maxPts), and the nodes on the way to that leaf that do not
// hold point i-1 are new at i: each point emits its nodes independently, in
// preorder.  Inputs with repeated points take the reference's sequential walk
// verbatim (a single-thread kernel), because its point bookkeeping then
// departs from the rule above.
//
// Balance (reference comboRipple, src/balance.cpp:801): the coarsest 2:1
// balanced refinement is unique.  With I_l the nodes at level l,
//   I_{l-1} = parent(input leaves at level l) U parents of the 3x3x3 blocks
//             around every q in I_l (8 octants per q, clipped to the domain).
// The sets grow in one hash table, level by level from the deepest, without
// a read-back between levels; one radix sort puts all nodes in preorder.
#include "dg_nodes.cuh"
#include "dg_walk.cuh"

#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <vector>

namespace dg {

// ------------------------------------------------------------------------
// quantize + Morton key (construct.cpp:930-942)
// ------------------------------------------------------------------------
// (unsigned int)(x * (double)(1u << D) / gLen): multiply, divide, truncate;
// valid iff the value before truncation lies in (-1, 2^D).  False otherwise.
//
// When gLen is a power of two 2^e (the unit cube of the workloads) both
// operations only move the exponent, so the value is x * 2^(D - e), truncated
// from the bits of x by integer shifts: GB300's narrow FP64 pipe, which the
// multiplications, comparisons and conversions of three coordinates kept busy,
// does nothing (16e6 points: 0.45 -> 0.37 ms).  Where x * 2^D would leave the
// normal range the value is 0 or out of the domain either way.
__device__ __forceinline__ bool quantize_pow2(double x, int shift, unsigned D, uint32_t &q) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52 & 0x7ffu) - 1023 + shift;  // |value| in [2^e, 2^(e+1)), or below 2^e for subnormals
  q = 0;
  if (e < 0) return true;  // in (-1, 1)
  if ((long long)b < 0 || e >= (int)D) return false;  // also infinities and NaN: e >= 1024 + shift > D
  q = (uint32_t)((b & 0xfffffffffffffull | 1ull << 52) >> (52 - e));
  return true;
}
__device__ __forceinline__ bool quantize_div(double x, double scale, double g, uint32_t &q) {
  const double v = __ddiv_rn(__dmul_rn(x, scale), g);
  q = 0;
  if (!(v > -1.0 && v < scale)) return false;
  q = (uint32_t)__double2uint_rz(v);
  return true;
}

// gx, gy, gz: the domain's lengths, or with POW2 the exponents D - e of the
// shifts.  vary collects the bits on which the keys differ from the first
// point's (two 64-bit words) where it is wanted.
template <bool POW2>
__global__ void k_quantize(const double *__restrict__ xyz, size_t n, double scale, double gx, double gy, double gz,
                           unsigned D, const uint64_t *__restrict__ seg_start, size_t nseg, Key128 *__restrict__ keys,
                           unsigned long long *__restrict__ vary, uint32_t *flags) {
  __shared__ Key128 first;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto key_of = [&](size_t j, bool &ok) {
    uint32_t u[3];
    ok = true;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double g = a == 0 ? gx : a == 1 ? gy : gz;
      if constexpr (POW2) ok = quantize_pow2(xyz[3 * j + a], (int)g, D, u[a]) && ok;
      else ok = quantize_div(xyz[3 * j + a], scale, g, u[a]) && ok;
    }
    if (!ok) u[0] = u[1] = u[2] = 0;
    return morton3(u[0], u[1], u[2]);
  };
  Key128 diff{0, 0};
  bool ok;
  if (vary) {
    if (threadIdx.x == 0) first = key_of(0, ok);
    __syncthreads();
  }
  if (i < n) {
    Key128 k = key_of(i, ok);
    if (!ok) set_flag(flags, DGF_DOMAIN);
    if (seg_start) {  // segment of point i: last s with seg_start[s] <= i
      size_t lo = 0, hi = nseg;
      while (hi - lo > 1) {
        size_t mid = (lo + hi) / 2;
        if (seg_start[mid] <= i) lo = mid;
        else hi = mid;
      }
      k = key_or(k, seg_key(lo, D));
    }
    keys[i] = make_tagged(k, D);
    if (vary) diff = key_xor(k, first);
  }
  if (vary) {
#pragma unroll
    for (int h = 0; h < 4; h++) {
      const uint64_t w = h < 2 ? diff.lo : diff.hi;
      const uint32_t v = __reduce_or_sync(0xffffffffu, (uint32_t)(h & 1 ? w >> 32 : w));
      if ((threadIdx.x & 31) == 0 && v) {
        const unsigned long long bits = (unsigned long long)v << (h & 1 ? 32 : 0);
        if (bits & ~__ldcg(vary + (h >> 1))) atomicOr(vary + (h >> 1), bits);
      }
    }
  }
}

// Orders runs of keys that agree above `begin` bits by the bits below, in
// place, one thread per run (an insertion sort); a run longer than RUN_MAX
// raises DGF_LONG_RUN.
constexpr int RUN_MAX = 32;
__global__ void k_sort_runs(Key128 *__restrict__ k, size_t n, unsigned begin, uint32_t *flags) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i + 1 >= n) return;
  const Key128 pre = key_shr(tag_anchor(k[i]), begin);
  if (!key_eq(key_shr(tag_anchor(k[i + 1]), begin), pre)) return;
  if (i > 0 && key_eq(key_shr(tag_anchor(k[i - 1]), begin), pre)) return;  // not the run's first
  size_t e = i + 2;
  while (e < n && e - i <= RUN_MAX && key_eq(key_shr(tag_anchor(k[e]), begin), pre)) e++;
  if (e - i > RUN_MAX) {
    set_flag(flags, DGF_LONG_RUN);
    return;
  }
  for (size_t a = i + 1; a < e; a++) {
    const Key128 v = k[a];
    size_t b = a;
    for (; b > i && key_lt(v, k[b - 1]); b--) k[b] = k[b - 1];
    k[b] = v;
  }
}

__device__ __forceinline__ unsigned leaf_level(const Key128 *__restrict__ p, size_t n, size_t i, unsigned m,
                                               unsigned D) {
  size_t lo = (i >= m) ? i - m : 0;
  size_t hi = (i + m < n) ? i : (n > m ? n - 1 - m : 0);
  int best = -1;
  if (n > m)
    for (size_t j = lo; j <= hi; j++) best = max(best, nca_level(p[j], p[j + m], D));
  return (unsigned)min(best + 1, (int)D);
}

// Node counts: point i adds the nodes on the way to its leaf (levels up to
// leaf level - 1) that do not hold point i-1, those below level NCA(i-1, i).
// path[i] = leaf level | (first new level) << 8, sums[b] = new nodes of block
// b's points; dupseg[s] = 1 where cloud s repeats a point (and 0x100 in
// flags); max_level = largest leaf level.
constexpr int P2O_BLOCK = 256, P2O_PER = 4, P2O_TILE = P2O_BLOCK * P2O_PER;
__global__ void __launch_bounds__(P2O_BLOCK) k_p2o_count(const Key128 *__restrict__ p, size_t n, unsigned m,
                                                         unsigned D, size_t nseg, uint16_t *__restrict__ path,
                                                         uint64_t *__restrict__ sums, uint32_t *__restrict__ dupseg,
                                                         unsigned long long *__restrict__ max_level, uint32_t *flags) {
  uint64_t total = 0;
  unsigned top = 0;
#pragma unroll
  for (int r = 0; r < P2O_PER; r++) {
    const size_t i = (size_t)blockIdx.x * P2O_TILE + r * P2O_BLOCK + threadIdx.x;
    if (i >= n) continue;
    const unsigned L = leaf_level(p, n, i, m, D);
    int a = -1;
    if (i > 0) {
      a = nca_level(p[i - 1], p[i], D);
      if (key_eq(p[i - 1], p[i])) {
        const uint64_t sg = seg_of(p[i], D);
        if (sg < nseg) dupseg[sg] = 1u;
        set_flag(flags, 0x100u);
      }
    }
    path[i] = (uint16_t)(L | (unsigned)(a + 1) << 8);
    if ((int)L > a + 1) total += L - (unsigned)(a + 1);
    top = max(top, L);
  }
  uint64_t sum;
  block_excl_scan<uint64_t, P2O_BLOCK>(total, sum);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && (unsigned long long)top > __ldcg(max_level)) atomicMax(max_level, (unsigned long long)top);
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
}

// the same for the leaves of a sorted octree: a leaf adds the nodes above it
// that do not hold its predecessor; leaves that are not aligned octants of the
// domain in strictly ascending order raise DGF_NOT_BALANCED
__global__ void __launch_bounds__(P2O_BLOCK) k_leaf_count(const Key128 *__restrict__ k, size_t n, unsigned D,
                                                          uint16_t *__restrict__ path, uint64_t *__restrict__ sums,
                                                          unsigned long long *__restrict__ max_level,
                                                          uint32_t *flags) {
  uint64_t total = 0;
  unsigned top = 0;
#pragma unroll
  for (int r = 0; r < P2O_PER; r++) {
    const size_t i = (size_t)blockIdx.x * P2O_TILE + r * P2O_BLOCK + threadIdx.x;
    if (i >= n) continue;
    const Key128 ki = k[i], a = tag_anchor(ki);
    const unsigned L = tag_level(ki);
    bool ok = L <= D && key_eq(morton_part(ki, D), a);
    if (ok && L < D) ok = key_eq(key_shl(key_shr(a, 3 * (D - L)), 3 * (D - L)), a);
    unsigned first = 0;
    if (i > 0) {
      const Key128 kp = k[i - 1];
      ok = ok && key_lt(tag_anchor(kp), a);
      first = min((unsigned)(nca_level(kp, ki, D) + 1), tag_level(kp));
    }
    if (!ok) set_flag(flags, DGF_NOT_BALANCED);
    path[i] = ok ? (uint16_t)(L | first << 8) : (uint16_t)0;
    if (ok && L > first) total += L - first;
    if (ok) top = max(top, L);
  }
  uint64_t sum;
  block_excl_scan<uint64_t, P2O_BLOCK>(total, sum);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && (unsigned long long)top > __ldcg(max_level)) atomicMax(max_level, (unsigned long long)top);
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
}

template <typename K>
__global__ void __launch_bounds__(P2O_BLOCK) k_p2o_nodes(const Key128 *__restrict__ p, size_t n, unsigned D,
                                                         unsigned Lm, const uint16_t *__restrict__ path,
                                                         const uint64_t *__restrict__ sums, K *__restrict__ out) {
  uint64_t at = sums[blockIdx.x];
#pragma unroll
  for (int r = 0; r < P2O_PER; r++) {
    const size_t i = (size_t)blockIdx.x * P2O_TILE + r * P2O_BLOCK + threadIdx.x;
    unsigned L = 0, l = 0;
    if (i < n) {
      L = path[i] & 255u;
      l = path[i] >> 8;
    }
    const uint32_t c = L > l ? L - l : 0u;
    uint32_t all;
    const uint32_t before = block_excl_scan<uint32_t, P2O_BLOCK>(c, all);
    if (c) {
      const Key128 a = tag_anchor(p[i]);
      for (uint64_t w = at + before; l < L; l++) out[w++] = node_of<K>(a, l, Lm, D);
    }
    at += all;
  }
}

// The leaves of the octrees whose nodes are given (sorted), 8 threads per
// node: child c of the node at index i is a leaf unless it is a node itself.
// The leaf's place is 7 (j - level) + digits + cloud, j the number of nodes
// before it in preorder (every cloud before it has one leaf more than 7 per
// node).  A warp holds four nodes and the 32 nodes that follow the first of
// them in its registers, so j comes from a search by shuffles; only a subtree
// that reaches past those is searched in memory.
// CHECK compares with the leaves that are there instead (DGF_NOT_BALANCED).
template <typename K, bool CHECK>
__global__ void __launch_bounds__(256) k_emit_leaves(const K *__restrict__ nodes, size_t nn, unsigned Lm, unsigned D,
                                                     Key128 *__restrict__ out, size_t total, uint32_t *flags) {
  typedef NodeWide<K> N;
  typedef typename N::W W;
  const int lane = threadIdx.x & 31;
  const size_t i0 = ((size_t)blockIdx.x * 256 + threadIdx.x) >> 5 << 2;  // the warp's first node
  if (i0 >= nn) return;
  const size_t i = i0 + (lane >> 3);
  const unsigned c = lane & 7;
  const W follow = i0 + 1 + lane < nn ? node_wide(nodes[i0 + 1 + lane]) : node_empty(W());
  const W k = i < nn ? node_wide(nodes[i]) : (W)0;
  const unsigned d = (unsigned)k & 31u;
  const W path = k >> 5;
  // child c, at depth D, and its key where it can be a node
  Key128 anchor;
  W ck = k + 1;  // level Lm: no node below
  if (d == Lm) {
    anchor = key_or(key_shl(N::key(path), 3 * (D - Lm)), key_shl(Key128{c, 0}, 3 * (D - Lm - 1)));
  } else {
    const W child = path + ((W)c << (3 * (Lm - d - 1)));
    anchor = key_shl(N::key(child), 3 * (D - Lm));
    ck = child << 5 | (W)(d + 1);
  }
  int at = 0;  // nodes of `follow` before ck
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (shfl_wide(follow, at + step - 1) < ck) at += step;
  const W found = shfl_wide(follow, at);
  if (i >= nn) return;
  size_t j = i0 + 1 + at;
  bool node = found == ck;
  if (at == 31 && found < ck) {  // galloping past the 32
    size_t lo = ++j, step = 1, hi;
    while (lo < nn && node_wide(nodes[lo]) < ck) {
      j = lo + 1;
      lo += step;
      step <<= 1;
    }
    hi = min(lo, nn);
    while (j < hi) {
      const size_t mid = j + (hi - j) / 2;
      if (node_wide(nodes[mid]) < ck) j = mid + 1;
      else hi = mid;
    }
    node = j < nn && node_wide(nodes[j]) == ck;
  }
  if (node && d != Lm) return;
  const W in_cloud = path & (((W)1 << (3 * Lm)) - 1);
  const size_t pos = 7 * (j - (d + 1)) + digit_sum(in_cloud) + c + (size_t)(path >> (3 * Lm));
  const Key128 leaf = make_tagged(anchor, d + 1);
  if constexpr (CHECK) {
    if (pos >= total || !key_eq(out[pos], leaf)) set_flag(flags, DGF_NOT_BALANCED);
  } else {
    if (pos < total) out[pos] = leaf;
  }
}

// per cloud: its first leaf's place, and its root where the root is a leaf
// (seg_off may be null)
template <typename K>
__global__ void k_emit_clouds(const K *__restrict__ nodes, size_t nn, unsigned Lm, unsigned D, size_t nseg,
                              Key128 *__restrict__ out, uint64_t *__restrict__ seg_off) {
  typedef typename NodeWide<K>::W W;
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s > nseg) return;
  size_t lo = 0, hi = nn;
  if (s == nseg) {
    lo = nn;
  } else {
    const W root = (W)s << (3 * Lm) << 5;
    while (lo < hi) {
      const size_t mid = lo + (hi - lo) / 2;
      if (node_wide(nodes[mid]) < root) lo = mid + 1;
      else hi = mid;
    }
    if (lo == nn || node_wide(nodes[lo]) != root) out[7 * lo + s] = make_tagged(seg_key(s, D), 0);
  }
  if (seg_off) seg_off[s] = 7 * lo + s;
}

// out's sorted nodes, taken over from a buffer
template <typename K>
static void keep_nodes(Octree &out, DBuf<K> &nodes, size_t nn, unsigned top) {
  out.nodes = nodes.release_ptr();
  out.n_node = nn;
  out.top = top;
  out.node_wide = sizeof(K) == 16;
}

// all leaves of nn sorted nodes of nseg clouds (7 nn + nseg octants)
template <typename K>
static void emit_octree(Context &ctx, const K *nodes, size_t nn, unsigned Lm, unsigned D, size_t nseg,
                        DBuf<Key128> &leaves, DBuf<uint64_t> &seg_off) {
  cudaStream_t s = ctx.stream;
  const size_t total = 7 * nn + nseg;
  leaves.alloc(total, s);
  if (nseg > 1) seg_off.alloc(nseg + 1, s);
  if (nseg > 1 || nn == 0) {
    ProfScope _prof(ctx, "emit_clouds", (double)nseg * 24);
    k_emit_clouds<K><<<grid_for(nseg + 1, 256), 256, 0, s>>>(nodes, nn, Lm, D, nseg, leaves.get(), seg_off.get());
    DG_LAUNCH_CHECK();
  }
  if (nn) {
    ProfScope _prof(ctx, "emit_leaves", (double)nn * sizeof(K) + (double)total * 16);
    k_emit_leaves<K, false><<<grid_for(8 * nn, 256), 256, 0, s>>>(nodes, nn, Lm, D, leaves.get(), total, nullptr);
    DG_LAUNCH_CHECK();
  }
}

__device__ __forceinline__ u128 kpos(Key128 k) { return to_u128(tag_anchor(k)); }

__device__ __forceinline__ int ctz128(u128 v) {
  uint64_t lo = (uint64_t)v;
  if (lo) return __ffsll((long long)lo) - 1;
  uint64_t hi = (uint64_t)(v >> 64);
  return hi ? 64 + __ffsll((long long)hi) - 1 : 128;
}
__device__ __forceinline__ int log2_128(u128 v) {  // v > 0
  uint64_t hi = (uint64_t)(v >> 64);
  if (hi) return 127 - __clzll((long long)hi);
  return 63 - __clzll((long long)(uint64_t)v);
}

// largest k <= D with s % 8^k == 0 and s + 8^k <= e (s < e); blocks never
// cross a cloud boundary because clouds are aligned 8^D ranges
__device__ __forceinline__ int block_exp(u128 s, u128 e, unsigned D) {
  int k1 = (s == 0) ? (int)D : min((int)D, ctz128(s) / 3);
  int k2 = log2_128(e - s) / 3;
  return min(k1, k2);
}

__device__ unsigned gap_count(u128 s, u128 e, unsigned D) {
  unsigned c = 0;
  while (s < e) {
    int k = block_exp(s, e, D);
    s += (u128)1 << (3 * k);
    c++;
  }
  return c;
}

__device__ size_t gap_emit(u128 s, u128 e, unsigned D, Key128 *out, size_t w) {
  while (s < e) {
    int k = block_exp(s, e, D);
    out[w++] = make_tagged(from_u128(s), D - (unsigned)k);
    s += (u128)1 << (3 * k);
  }
  return w;
}

__device__ __forceinline__ u128 seed_end(Key128 s, unsigned D) {
  return kpos(s) + ((u128)1 << (3 * (D - tag_level(s))));
}

__global__ void k_fill_count(const Key128 *__restrict__ seeds, size_t ns, unsigned D, u128 total,
                             uint32_t *__restrict__ cnt) {
  size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  u128 e = (j + 1 < ns) ? kpos(seeds[j + 1]) : total;
  unsigned c = 1 + gap_count(seed_end(seeds[j], D), e, D);
  if (j == 0) c += gap_count(0, kpos(seeds[0]), D);
  cnt[j] = c;
}

__global__ void k_fill_emit(const Key128 *__restrict__ seeds, size_t ns, unsigned D, u128 total,
                            const uint64_t *__restrict__ off, Key128 *__restrict__ out) {
  size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  size_t w = off[j];
  if (j == 0) w = gap_emit(0, kpos(seeds[0]), D, out, w);
  out[w++] = seeds[j];
  u128 e = (j + 1 < ns) ? kpos(seeds[j + 1]) : total;
  gap_emit(seed_end(seeds[j], D), e, D, out, w);
}

// ------------------------------------------------------------------------
// the reference walk for clouds with repeated points (dg_walk.cuh): one
// block per such cloud, thread 0 walks it; count pass then emit pass
// ------------------------------------------------------------------------
__global__ void k_p2o_walk_segments(const Key128 *__restrict__ pk, const uint64_t *__restrict__ pt_start,
                                    const uint32_t *__restrict__ dup_list, unsigned m, unsigned D,
                                    const uint64_t *__restrict__ out_off, Key128 *__restrict__ out,
                                    unsigned long long *counts, bool batched) {
  if (threadIdx.x != 0) return;
  const uint32_t s = dup_list[blockIdx.x];
  const size_t b = pt_start[s], e = pt_start[s + 1];
  bool outside = false;
  size_t c = p2o_walk(pk + b, e - b, m, D, out ? out + out_off[blockIdx.x] : nullptr, seg_key(s, D), &outside);
  counts[blockIdx.x] = c;
  if (outside && batched) counts[blockIdx.x] = (unsigned long long)P2O_WALK_OUTSIDE;
}

// place each cloud's octants at their final offsets: clouds with repeated
// points take the walk's output, the others the parallel construction's.
// The walk outputs are stored cloud after cloud in dup-list order; a walk
// octant's cloud is found from its position (its key may lie outside the
// cloud's domain, see dg_walk.cuh).
__global__ void k_assemble(const Key128 *__restrict__ par, size_t npar, const uint64_t *__restrict__ par_off,
                           const Key128 *__restrict__ walk, const uint64_t *__restrict__ walk_off, size_t nd,
                           const uint32_t *__restrict__ dup_list, const uint32_t *__restrict__ dupseg, size_t nseg,
                           const uint64_t *__restrict__ final_off, unsigned D, Key128 *__restrict__ out,
                           size_t nwalk_total) {
  size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < npar) {
    uint64_t s = seg_of(par[j], D);
    if (s < nseg && !dupseg[s]) out[final_off[s] + (j - par_off[s])] = par[j];
  }
  if (j < nwalk_total) {
    size_t lo = 0, hi = nd;  // last slot with walk_off[slot] <= j
    while (hi - lo > 1) {
      size_t mid = (lo + hi) / 2;
      if (walk_off[mid] <= j) lo = mid;
      else hi = mid;
    }
    uint32_t s = dup_list[lo];
    out[final_off[s] + (j - walk_off[lo])] = walk[j];
  }
}

// ------------------------------------------------------------------------
// host: point sort and construction
// ------------------------------------------------------------------------
void check_device_flags(Context &ctx, const char *where) {
  uint32_t f = read_scalar(ctx, ctx.d_flags);
  if (f) {
    DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), ctx.stream));
    if (f & DGF_DOMAIN) fail(DG_ERR_DOMAIN, std::string(where) + ": input outside the domain");
    if (f & DGF_NOT_BALANCED) fail(DG_ERR_NOT_BALANCED, std::string(where) + ": input is not a complete 2:1 balanced octree");
    if (f & DGF_TIMEOUT) fail(DG_ERR_TIMEOUT, std::string(where) + ": a device wait timed out");
    if (f & DGF_INTERNAL) fail(DG_ERR_INTERNAL, std::string(where) + ": internal consistency check failed");
    if (f & DGF_ORDER) fail(DG_ERR_INVALID_ARG, std::string(where) + ": input is not sorted / unique as declared");
  }
}

// The points as sorted tagged keys.  LSD passes over all 3D key bits cost 12
// reads and writes of the keys, while log2(n) + PREFIX_EXTRA leading bits
// leave few points together: only those are sorted (5 passes for 16e6
// points), from the highest bit on which the keys differ (read back for large
// inputs, where the wait costs little), and k_sort_runs orders the short runs
// left.  With `full` every bit is sorted: the caller's answer to
// DGF_LONG_RUN (points clustered within a few tiny cells).  ctx.d_flags
// collects what the kernels raise; sorted_flags() reads it.
constexpr int PREFIX_EXTRA = 16;
constexpr size_t VARY_MIN = size_t(1) << 18;

// flags raised by quantize_sorted's kernels, after a wait for the stream;
// throws on all but DGF_LONG_RUN and the repeated-points bit
static uint32_t sorted_flags(Context &ctx) {
  const uint32_t f = read_scalar(ctx, ctx.d_flags), keep = DGF_LONG_RUN | 0x100u;
  if (f & ~keep) check_device_flags(ctx, "points2Octree");
  if (f) DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), ctx.stream));
  return f;
}

static Key128 *quantize_sorted(Context &ctx, const double *d_xyz, size_t n, const double g[3], unsigned D,
                               const uint64_t *d_seg_start, size_t nseg, unsigned seg_bits, bool full,
                               DBuf<Key128> &keys, DBuf<Key128> &tmp) {
  cudaStream_t s = ctx.stream;
  keys.alloc(n, s);
  tmp.alloc(n, s);
  unsigned long long *d_vary = n >= VARY_MIN && !full ? ctx.d_scratch + 4 : nullptr;
  DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
  if (d_vary) DG_CUDA(cudaMemsetAsync(d_vary, 0, 2 * sizeof(unsigned long long), s));
  {
    ProfScope _prof(ctx, "quantize", (double)n * 40);
    // e where v = 2^e, else INT_MIN
    auto pow2 = [](double v) {
      int e = 0;
      return std::frexp(v, &e) == 0.5 && e > -900 && e < 900 ? e - 1 : INT_MIN;
    };
    const int e[3] = {pow2(g[0]), pow2(g[1]), pow2(g[2])};
    if (e[0] != INT_MIN && e[1] != INT_MIN && e[2] != INT_MIN)
      k_quantize<true><<<grid_for(n, 256), 256, 0, s>>>(d_xyz, n, 0.0, (double)((int)D - e[0]),
                                                        (double)((int)D - e[1]), (double)((int)D - e[2]), D,
                                                        d_seg_start, nseg, keys.get(), d_vary, ctx.d_flags);
    else
      k_quantize<false><<<grid_for(n, 256), 256, 0, s>>>(d_xyz, n, (double)(1u << D), g[0], g[1], g[2], D, d_seg_start,
                                                         nseg, keys.get(), d_vary, ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  int hi = 3 * (int)D + (int)seg_bits;
  if (d_vary) {
    DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_vary, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    sorted_flags(ctx);
    const unsigned long long lo = ctx.h_scratch[4], up = ctx.h_scratch[5];
    const int bits = up ? 128 - __builtin_clzll(up) : lo ? 64 - __builtin_clzll(lo) : 0;
    hi = std::min(hi, bits);
  }
  int want = PREFIX_EXTRA;
  while (want < 63 && ((size_t)1 << (want - PREFIX_EXTRA)) < n) want++;
  const int begin = full ? 0 : std::max(0, hi - (want + 7) / 8 * 8);
  Key128 *sorted = radix_sort<Key128>(ctx, keys.get(), tmp.get(), n, hi, begin);
  if (begin > 0) {
    ProfScope _prof(ctx, "sort_runs", (double)n * 16);
    k_sort_runs<<<grid_for(n, 256), 256, 0, s>>>(sorted, n, (unsigned)begin, ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  return sorted;
}

size_t sort_points(Context &ctx, const double *d_xyz, size_t n, const double g[3], unsigned D, Key128 *d_out,
                   bool *has_dups) {
  if (n == 0) return 0;
  DBuf<Key128> keys, tmp;
  Key128 *sorted = quantize_sorted(ctx, d_xyz, n, g, D, nullptr, 1, 0, false, keys, tmp);
  if (sorted_flags(ctx) & DGF_LONG_RUN) {
    sorted = quantize_sorted(ctx, d_xyz, n, g, D, nullptr, 1, 0, true, keys, tmp);
    sorted_flags(ctx);
  }
  DBuf<uint32_t> flags(n, ctx.stream);
  {
    ProfScope _prof(ctx, "flag_unique", (double)n * 20);
    k_flag_unique<Key128><<<grid_for(n, 256), 256, 0, ctx.stream>>>(sorted, n, flags.get());
    DG_LAUNCH_CHECK();
  }
  size_t nu = compact<Key128>(ctx, sorted, flags.get(), n, d_out);
  if (has_dups) *has_dups = nu != n;
  return nu;
}

void points_to_octree(Context &ctx, const double *d_xyz, size_t n, const double g[3], unsigned D, unsigned m,
                      Octree &out, const uint64_t *h_seg_start, size_t nseg) {
  if (m == 0 || D > 30) fail(DG_ERR_INVALID_ARG, "points2Octree: maxNumPts must be >= 1 and maxDepth <= 30");
  if (n >= 0x7fffffffull) fail(DG_ERR_INVALID_ARG, "points2Octree: too many points");
  if (nseg == 0) fail(DG_ERR_INVALID_ARG, "points2Octree: no clouds");
  const unsigned SB = bits_for(nseg);
  if (3 * D + SB > 120) fail(DG_ERR_INVALID_ARG, "points2Octree: too many clouds for maxDepth");
  if (h_seg_start) {
    if (h_seg_start[0] != 0 || h_seg_start[nseg] != n)
      fail(DG_ERR_INVALID_ARG, "points2Octree: cloud offsets must run from 0 to n");
    for (size_t s = 0; s < nseg; s++)
      if (h_seg_start[s + 1] < h_seg_start[s]) fail(DG_ERR_INVALID_ARG, "points2Octree: cloud offsets decrease");
  }
  out.max_depth = D;
  out.nseg = nseg;
  out.seg_bits = SB;
  cudaStream_t s = ctx.stream;
  const u128 total = (u128)nseg << (3 * D);
  DBuf<uint64_t> d_seg_start;
  if (nseg > 1) {
    d_seg_start.alloc(nseg + 1, s);
    DG_CUDA(cudaMemcpyAsync(d_seg_start.get(), h_seg_start, (nseg + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  }
  if (D == 0 || n == 0 || (nseg == 1 && n <= m)) {
    // construct.cpp:916-920, 948-952: a cloud with at most maxPts points is
    // the root alone (still validate the points like the quantize loop)
    if (n && D) {
      DBuf<Key128> keys(n, s);
      {
        ProfScope _prof(ctx, "quantize", (double)n * 40);
        k_quantize<false><<<grid_for(n, 256), 256, 0, s>>>(d_xyz, n, (double)(1u << D), g[0], g[1], g[2], D, nullptr,
                                                           1, keys.get(), nullptr, ctx.d_flags);
        DG_LAUNCH_CHECK();
      }
      check_device_flags(ctx, "points2Octree");
    }
    std::vector<Key128> roots(nseg);
    for (size_t i = 0; i < nseg; i++) roots[i] = make_tagged(seg_key(i, D), 0);
    out.n = nseg;
    DG_CUDA(cudaMallocAsync((void **)&out.keys, nseg * sizeof(Key128), s));
    DG_CUDA(cudaMemcpyAsync(out.keys, roots.data(), nseg * sizeof(Key128), cudaMemcpyHostToDevice, s));
    if (nseg > 1) {
      std::vector<uint64_t> off(nseg + 1);
      for (size_t i = 0; i <= nseg; i++) off[i] = i;
      DG_CUDA(cudaMallocAsync((void **)&out.seg_off, (nseg + 1) * sizeof(uint64_t), s));
      DG_CUDA(cudaMemcpyAsync(out.seg_off, off.data(), (nseg + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
    }
    DG_CUDA(cudaStreamSynchronize(s));
    return;
  }
  DBuf<Key128> keys, tmp;
  Key128 *p = nullptr;
  const size_t nblocks = (n + P2O_TILE - 1) / P2O_TILE;
  DBuf<uint32_t> dupseg(nseg, s);  // clouds with repeated points
  DBuf<uint16_t> path(n, s);
  DBuf<uint64_t> sums(nblocks, s);
  unsigned long long *d_info = ctx.d_scratch;  // {nodes, largest leaf level}
  uint32_t dupflag = 0;
  for (bool full : {false, true}) {
    p = quantize_sorted(ctx, d_xyz, n, g, D, d_seg_start.get(), nseg, SB, full, keys, tmp);
    DG_CUDA(cudaMemsetAsync(dupseg.get(), 0, nseg * sizeof(uint32_t), s));
    DG_CUDA(cudaMemsetAsync(d_info, 0, 2 * sizeof(unsigned long long), s));
    {
      ProfScope _prof(ctx, "p2o_count", (double)n * 18);
      k_p2o_count<<<(unsigned)nblocks, P2O_BLOCK, 0, s>>>(p, n, m, D, nseg, path.get(), sums.get(), dupseg.get(),
                                                          d_info + 1, ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    exclusive_scan<uint64_t, uint64_t>(sums.get(), sums.get(), nblocks, reinterpret_cast<uint64_t *>(d_info), s);
    DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_info, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    const uint32_t f = sorted_flags(ctx);
    dupflag = f & 0x100u;
    if (!(f & DGF_LONG_RUN)) break;
  }
  const size_t nn = (size_t)ctx.h_scratch[4];
  const unsigned top = std::max(1u, (unsigned)ctx.h_scratch[5]);  // deepest leaf level

  // parallel construction over all points (clouds with repeated points are
  // replaced below): the nodes in preorder, then their leaves
  DBuf<Key128> res;
  DBuf<uint64_t> seg_off;
  auto construct = [&](auto tag) {
    typedef decltype(tag) K;
    DBuf<K> nodes(nn ? nn : 1, s);
    {
      ProfScope _prof(ctx, "p2o_nodes", (double)n * 18 + (double)nn * sizeof(K));
      k_p2o_nodes<K><<<(unsigned)nblocks, P2O_BLOCK, 0, s>>>(p, n, D, top - 1, path.get(), sums.get(), nodes.get());
      DG_LAUNCH_CHECK();
    }
    emit_octree<K>(ctx, nodes.get(), nn, top - 1, D, nseg, res, seg_off);
    if (!dupflag) keep_nodes(out, nodes, nn, top);
  };
  if (nodes_fit_64(top, SB)) construct(uint64_t());
  else construct(Key128());
  const size_t npar = 7 * nn + nseg;
  if (!dupflag) {
    out.n = npar;
    out.keys = res.release_ptr();
    out.seg_off = nseg > 1 ? seg_off.release_ptr() : nullptr;
    DG_CUDA(cudaStreamSynchronize(s));
    return;
  }

  // walk every cloud with repeated points
  std::vector<uint32_t> h_dup(nseg);
  DG_CUDA(cudaMemcpyAsync(h_dup.data(), dupseg.get(), nseg * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  std::vector<uint64_t> h_par_off(nseg + 1);
  if (nseg == 1) {
    seg_off.alloc(2, s);
    const uint64_t one[2] = {0, npar};
    DG_CUDA(cudaMemcpyAsync(seg_off.get(), one, sizeof(one), cudaMemcpyHostToDevice, s));
  }
  DG_CUDA(cudaMemcpyAsync(h_par_off.data(), seg_off.get(), (nseg + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  DG_CUDA(cudaStreamSynchronize(s));
  std::vector<uint32_t> dup_list, walk_slot(nseg, 0xffffffffu);
  for (size_t i = 0; i < nseg; i++)
    if (h_dup[i]) {
      walk_slot[i] = (uint32_t)dup_list.size();
      dup_list.push_back((uint32_t)i);
    }
  const size_t nd = dup_list.size();
  std::vector<uint64_t> h_pt_start(nseg + 1);
  if (h_seg_start) {
    for (size_t i = 0; i <= nseg; i++) h_pt_start[i] = h_seg_start[i];
  } else {
    h_pt_start[0] = 0;
    h_pt_start[1] = n;
  }
  DBuf<uint64_t> d_pt_start(nseg + 1, s), d_walk_off(nd + 1, s);
  DBuf<uint32_t> d_dup_list(nd, s);
  DBuf<unsigned long long> d_counts(nd, s);
  DG_CUDA(cudaMemcpyAsync(d_pt_start.get(), h_pt_start.data(), (nseg + 1) * 8, cudaMemcpyHostToDevice, s));
  DG_CUDA(cudaMemcpyAsync(d_dup_list.get(), dup_list.data(), nd * 4, cudaMemcpyHostToDevice, s));
  {
    ProfScope _prof(ctx, "p2o_walk_serial", (double)n * 16);
    k_p2o_walk_segments<<<(unsigned)nd, 32, 0, s>>>(p, d_pt_start.get(), d_dup_list.get(), m, D, nullptr, nullptr,
                                                    d_counts.get(), nseg > 1);
    DG_LAUNCH_CHECK();
  }
  std::vector<unsigned long long> h_counts(nd);
  DG_CUDA(cudaMemcpyAsync(h_counts.data(), d_counts.get(), nd * 8, cudaMemcpyDeviceToHost, s));
  DG_CUDA(cudaStreamSynchronize(s));
  std::vector<uint64_t> h_walk_off(nd + 1, 0);
  for (size_t i = 0; i < nd; i++) {
    if (h_counts[i] == (unsigned long long)P2O_WALK_NO_END)
      fail(DG_ERR_INVALID_ARG,
           "points2Octree: with these repeated points the reference construction walk never terminates");
    if (h_counts[i] == (unsigned long long)P2O_WALK_OUTSIDE)
      fail(DG_ERR_DOMAIN,
           "points2Octree: with these repeated points the reference construction emits octants outside the domain, "
           "which a batch can not hold (build this cloud alone)");
    h_walk_off[i + 1] = h_walk_off[i] + h_counts[i];
  }
  const size_t nwalk = h_walk_off[nd];
  DG_CUDA(cudaMemcpyAsync(d_walk_off.get(), h_walk_off.data(), (nd + 1) * 8, cudaMemcpyHostToDevice, s));
  DBuf<Key128> walk_out(nwalk ? nwalk : 1, s);
  {
    ProfScope _prof(ctx, "p2o_walk_serial", (double)n * 16 + (double)nwalk * 16);
    k_p2o_walk_segments<<<(unsigned)nd, 32, 0, s>>>(p, d_pt_start.get(), d_dup_list.get(), m, D, d_walk_off.get(),
                                                    walk_out.get(), d_counts.get(), nseg > 1);
    DG_LAUNCH_CHECK();
  }
  // final offsets
  std::vector<uint64_t> h_final(nseg + 1, 0);
  for (size_t i = 0; i < nseg; i++) {
    uint64_t c = h_dup[i] ? h_counts[walk_slot[i]] : (h_par_off[i + 1] - h_par_off[i]);
    h_final[i + 1] = h_final[i] + c;
  }
  const size_t nfinal = h_final[nseg];
  DBuf<uint64_t> d_final(nseg + 1, s);
  DG_CUDA(cudaMemcpyAsync(d_final.get(), h_final.data(), (nseg + 1) * 8, cudaMemcpyHostToDevice, s));
  DBuf<Key128> fin(nfinal ? nfinal : 1, s);
  {
    ProfScope _prof(ctx, "p2o_assemble", (double)(npar + nwalk) * 32);
    k_assemble<<<grid_for(std::max(npar, nwalk), 256), 256, 0, s>>>(res.get(), npar, seg_off.get(), walk_out.get(),
                                                                    d_walk_off.get(), nd, d_dup_list.get(),
                                                                    dupseg.get(), nseg, d_final.get(), D, fin.get(),
                                                                    nwalk);
    DG_LAUNCH_CHECK();
  }
  out.n = nfinal;
  out.keys = fin.release_ptr();
  if (nseg > 1) {
    out.seg_off = d_final.release_ptr();
  }
  DG_CUDA(cudaStreamSynchronize(s));
}

bool octree_nodes(Context &ctx, const Octree &in, Octree &out) {
  cudaStream_t s = ctx.stream;
  const size_t n = in.n, nblocks = (n + P2O_TILE - 1) / P2O_TILE;
  const unsigned D = in.max_depth;
  out = Octree();
  out.max_depth = D;
  out.n = n;
  if (in.nseg != 1) fail(DG_ERR_UNSUPPORTED, "octree: one cloud per call");
  auto in_order = [&] {
    const uint32_t f = read_scalar(ctx, ctx.d_flags);
    if (f & ~(uint32_t)DGF_NOT_BALANCED) check_device_flags(ctx, "octree");
    if (f) DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
    return f == 0;
  };
  DBuf<uint16_t> path(n, s);
  DBuf<uint64_t> sums(nblocks, s);
  unsigned long long *d_info = ctx.d_scratch;  // {nodes, deepest leaf level}
  DG_CUDA(cudaMemsetAsync(d_info, 0, 2 * sizeof(unsigned long long), s));
  DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
  {
    ProfScope _prof(ctx, "leaf_count", (double)n * 18);
    k_leaf_count<<<(unsigned)nblocks, P2O_BLOCK, 0, s>>>(in.keys, n, D, path.get(), sums.get(), d_info + 1,
                                                         ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  exclusive_scan<uint64_t, uint64_t>(sums.get(), sums.get(), nblocks, reinterpret_cast<uint64_t *>(d_info), s);
  DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_info, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  if (!in_order()) return false;
  const size_t nn = (size_t)ctx.h_scratch[4];
  const unsigned top = (unsigned)ctx.h_scratch[5];
  if (!nn || n != 7 * nn + 1) return false;
  auto make = [&](auto tag) {
    typedef decltype(tag) K;
    DBuf<K> nodes(nn, s);
    k_p2o_nodes<K><<<(unsigned)nblocks, P2O_BLOCK, 0, s>>>(in.keys, n, D, top - 1, path.get(), sums.get(), nodes.get());
    DG_LAUNCH_CHECK();
    k_emit_leaves<K, true><<<grid_for(8 * nn, 256), 256, 0, s>>>(nodes.get(), nn, top - 1, D, in.keys, n, ctx.d_flags);
    DG_LAUNCH_CHECK();
    if (!in_order()) return false;
    keep_nodes(out, nodes, nn, top);
    return true;
  };
  return nodes_fit_64(top, 0) ? make(uint64_t()) : make(Key128());
}

void octree_segment_offsets(Context &ctx, const Octree &o, uint64_t *h_off) {
  if (o.nseg == 1 || !o.seg_off) {
    h_off[0] = 0;
    h_off[1] = o.n;
    return;
  }
  DG_CUDA(cudaMemcpyAsync(h_off, o.seg_off, (o.nseg + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
  DG_CUDA(cudaStreamSynchronize(ctx.stream));
}

// ------------------------------------------------------------------------
// balance
// ------------------------------------------------------------------------
// Flags octants that are not aligned octants of the domain of their cloud
// (the reference asserts on those, octFunctions.cpp:310) and counts, per level
// of the parent, the leaves that bring a parent: all but those whose
// predecessor has the same one.
__device__ __forceinline__ bool brings_parent(const Key128 *__restrict__ k, size_t i, Key128 ki, unsigned D) {
  const unsigned l = tag_level(ki);
  if (l == 0) return false;
  if (i == 0) return true;
  const Key128 kp = k[i - 1];
  const unsigned sh = 3 * (D - l + 1);
  return !(tag_level(kp) == l && key_eq(key_shr(tag_anchor(kp), sh), key_shr(tag_anchor(ki), sh)));
}

__global__ void k_bal_scan(const Key128 *__restrict__ k, size_t n, unsigned D, uint64_t nseg,
                           unsigned long long *hist, uint32_t *flags) {
  __shared__ unsigned int h[32];
  if (threadIdx.x < 32) h[threadIdx.x] = 0;
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const Key128 ki = k[i];
    const unsigned l = tag_level(ki);
    const Key128 a = morton_part(ki, D);
    bool ok = l <= D && seg_of(ki, D) < nseg;
    if (ok && l < D) ok = key_eq(key_shl(key_shr(a, 3 * (D - l)), 3 * (D - l)), a);
    if (!ok) atomicOr(flags, DGF_DOMAIN);
    else if (brings_parent(k, i, ki, D)) atomicAdd(&h[l - 1], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32 && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

// Where the nodes go: those the balance starts from at off[l] of `start`, level
// by level; the grown ones in the order of their making in `grown`.  Counters
// on the device: room per level, nodes per level from the start, and grown.
struct BalCounts {
  unsigned long long room[32], start[32], grown[32];
};
__device__ __forceinline__ unsigned long long bal_off(const BalCounts *__restrict__ cnt, unsigned l) {
  unsigned long long at = 0;
  for (unsigned q = 0; q < l; q++) at += cnt->room[q];
  return at;
}

// nodes per level of an octree that has them
template <typename K>
__global__ void k_bal_node_levels(const K *__restrict__ nodes, size_t nn, unsigned long long *__restrict__ hist) {
  __shared__ unsigned h[32];
  if (threadIdx.x < 32) h[threadIdx.x] = 0;
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += (size_t)gridDim.x * blockDim.x)
    atomicAdd(&h[(unsigned)node_wide(nodes[i]) & 31u], 1u);
  __syncthreads();
  if (threadIdx.x < 32 && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

// the nodes that the balance starts from into the table and their level's
// list: the input's own (sorted) nodes, or with LEAVES the parents of its leaves
template <typename K, bool LEAVES>
__global__ void __launch_bounds__(256) k_bal_start(const void *__restrict__ in, size_t n, unsigned D, unsigned Lm,
                                                   K *__restrict__ tab, uint64_t mask, K *__restrict__ list,
                                                   size_t room, BalCounts *__restrict__ cnt, uint32_t *flags) {
  __shared__ unsigned num[32];
  __shared__ unsigned long long base[32];
  if (threadIdx.x < 32) num[threadIdx.x] = 0;
  __syncthreads();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  bool won = false;
  K key{};
  unsigned l = 0, rank = 0;
  if (i < n) {
    if constexpr (LEAVES) {
      const Key128 *k = static_cast<const Key128 *>(in);
      const Key128 ki = k[i];
      won = brings_parent(k, i, ki, D);
      if (won) {
        l = tag_level(ki) - 1;
        key = node_of<K>(tag_anchor(ki), l, Lm, D);
      }
    } else {
      key = static_cast<const K *>(in)[i];
      l = (unsigned)node_wide(key) & 31u;
      won = true;
    }
    if (won) won = node_insert<K>(tab, mask, node_wide(key), Lm, flags);
    if (won) rank = atomicAdd(&num[l], 1u);
  }
  __syncwarp();
  __syncthreads();
  if (threadIdx.x < 32 && num[threadIdx.x])
    base[threadIdx.x] =
        bal_off(cnt, threadIdx.x) + atomicAdd(&cnt->start[threadIdx.x], (unsigned long long)num[threadIdx.x]);
  __syncthreads();
  if (!won) return;
  if (base[l] + rank < room) list[base[l] + rank] = key;
  else set_flag(flags, DGF_INTERNAL);
}

// One level of the recursion: for every node q of level l the 8 parents (level
// l - 1) of q's 3x3x3 block that lie in the domain.  Without corners
// (balanceOctree's incCorner = false: faces and edges only, the 18 directions
// of TreeNode::addBalancingDescendants, src/TreeNode.cpp:160-190) not the
// parent that only q's corner neighbours reach (outward on all three axes).
// A block takes 256 nodes at a time; its 2048 candidates are made unique in
// shared memory first (the nodes of a block lie close together, and 3 of 4
// candidates repeat), so the table in L2 sees each once per block.
constexpr int BAL_TILE = 256, BAL_CAND = 8 * BAL_TILE, BAL_SLOTS = 2 * BAL_CAND;
constexpr uint32_t BAL_FREE = 0xffffffffu;
template <typename K>
struct BalSmem {
  K cand[BAL_CAND];
  uint32_t slot[BAL_SLOTS];
  uint16_t list[BAL_CAND], won[BAL_CAND];
  unsigned n_cand, n_won;
  unsigned long long at;
};

// appends v of the lanes that say so to a list in shared memory.  All lanes of
// the warp take part, which brings them together after the diverging probes and
// before the block's next barrier.  With each lane adding to the counter where
// it left its probes, balances of 1.4e8 nodes with 128-bit keys at times lost or
// repeated a few; why is not established (the barrier alone orders the writes
// before the reads).  So entries are checked before they are used as indices,
// and the sorted list of all nodes by k_bal_check.
__device__ __forceinline__ void warp_append(bool mine, uint16_t v, unsigned *n, uint16_t *list) {
  const unsigned m = __ballot_sync(0xffffffffu, mine);
  if (!m) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  unsigned at = 0;
  if (lane == leader) at = atomicAdd(n, (unsigned)__popc(m));
  at = __shfl_sync(0xffffffffu, at, leader);
  if (mine) list[at + __popc(m & ((1u << lane) - 1u))] = v;
  __syncwarp();
}

template <typename K>
__global__ void __launch_bounds__(BAL_TILE) k_bal_level(unsigned l, unsigned Lm, bool inc_corner, K *__restrict__ tab,
                                                        uint64_t mask, const K *__restrict__ start,
                                                        K *grown, size_t grown_cap, BalCounts *__restrict__ cnt,
                                                        uint32_t *flags) {
  typedef NodeWide<K> N;
  typedef typename N::W W;
  extern __shared__ __align__(16) unsigned char bal_raw[];
  BalSmem<K> &S = *reinterpret_cast<BalSmem<K> *>(bal_raw);
  const int t = threadIdx.x;
  const size_t n0 = cnt->start[l], n1 = cnt->grown[l], off = bal_off(cnt, l);
  size_t first = 0;  // grown nodes of the levels below
  for (unsigned q = l + 1; q <= Lm; q++) first += cnt->grown[q];
  if (first + n1 > grown_cap) return;  // the list overflowed (flagged): the host starts again
  const size_t n = n0 + n1, next = first + n1;
  // nodes per tile: all blocks get some, up to BAL_TILE
  const unsigned per = (unsigned)min((size_t)BAL_TILE, max((size_t)16, (n + gridDim.x - 1) / gridDim.x));
  unsigned slots = 32;
  while (slots < 16 * per) slots <<= 1;
  for (size_t base = (size_t)blockIdx.x * per; base < n; base += (size_t)gridDim.x * per) {
    const unsigned here = (unsigned)min((size_t)per, n - base);
    for (unsigned q = t; q < slots; q += BAL_TILE) S.slot[q] = BAL_FREE;
    if (t == 0) S.n_cand = S.n_won = 0;
    if (t < here) {
      const size_t i = base + t;
      const W k = node_wide(i < n0 ? start[off + i] : grown[first + (i - n0)]);
      const W path = k >> 5;
      const W cloud = path >> (3 * Lm);
      const W idx = (path & (((W)1 << (3 * Lm)) - 1)) >> (3 * (Lm - l));
      uint32_t c[3];
      demorton3(N::key(idx), c[0], c[1], c[2]);  // level-l integer coordinates
      const uint32_t side = 1u << (l - 1);  // parents per axis
      uint32_t opt[3][2];
      bool in[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        opt[a][0] = c[a] >> 1;
        opt[a][1] = (c[a] & 1u) ? opt[a][0] + 1 : opt[a][0] - 1;
        in[a] = opt[a][1] < side;  // -1 wraps round
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const bool skip = ((q & 1) && !in[0]) || ((q & 2) && !in[1]) || ((q & 4) && !in[2]) || (q == 7 && !inc_corner);
        const W par = cloud << (3 * (l - 1)) | N::of(morton3(opt[0][q & 1], opt[1][q >> 1 & 1], opt[2][q >> 2]));
        S.cand[8 * t + q] = skip ? N::narrow(node_empty(k)) : N::narrow(par << (3 * (Lm - l + 1)) << 5 | (W)(l - 1));
      }
    }
    __syncthreads();
    for (unsigned r = 0; r < 8 * here; r += BAL_TILE) {
      const unsigned me = r + t;
      bool mine = false;
      const W key = me < 8 * here ? node_wide(S.cand[me]) : node_empty(W());
      if (key != node_empty(key)) {
        const uint64_t hash = node_hash(key, Lm);
        uint32_t h = (uint32_t)(hash ^ hash >> 24) & (slots - 1);
        for (unsigned probe = 0; probe < slots; probe++) {
          const uint32_t cur = atomicCAS(&S.slot[h], BAL_FREE, me);
          mine = cur == BAL_FREE;
          if (mine || node_wide(S.cand[cur]) == key) break;
          h = (h + 1) & (slots - 1);
        }
      }
      warp_append(mine, (uint16_t)me, &S.n_cand, S.list);
    }
    __syncthreads();
    const unsigned nc = S.n_cand;
    for (unsigned r = 0; r < nc; r += BAL_TILE) {
      const unsigned q = r + t, me = q < nc ? S.list[q] : 0u;
      const bool ok = q < nc && me < 8 * here;
      if (q < nc && !ok) set_flag(flags, DGF_INTERNAL);
      const bool won = ok && node_insert<K>(tab, mask, node_wide(S.cand[me]), Lm, flags);
      warp_append(won, (uint16_t)me, &S.n_won, S.won);
    }
    __syncthreads();
    const unsigned nw = S.n_won;
    if (t == 0 && nw) S.at = next + atomicAdd(&cnt->grown[l - 1], (unsigned long long)nw);
    __syncthreads();
    for (unsigned q = t; q < nw; q += BAL_TILE) {
      const unsigned me = S.won[q];
      if (me >= 8 * here) set_flag(flags, DGF_INTERNAL);
      else if (S.at + q < grown_cap) grown[S.at + q] = S.cand[me];
      else set_flag(flags, DGF_CAPACITY);
    }
    __syncthreads();
  }
}

// all nodes side by side: the start's lists without the room their repeats
// left, then the grown ones
struct BalGather {
  unsigned long long off[32], num[32], to[32];
};
template <typename K>
__global__ void k_bal_gather(const K *__restrict__ start, BalGather g, size_t n_room, K *__restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_room) return;
  int l = 0;
  while (l < 31 && i >= g.off[l + 1]) l++;
  const size_t r = i - g.off[l];
  if (r < g.num[l]) out[g.to[l] + r] = start[i];
}

// the sorted nodes as an octree's: neighbours that do not follow one another
// raise DGF_INTERNAL.  Four per thread, loaded together (1.25e7 nodes: 27 us, 43
// with one).
constexpr int CHECK_PER = 4;
template <typename K>
__global__ void __launch_bounds__(256) k_bal_check(const K *__restrict__ nodes, size_t nn, unsigned Lm,
                                                   uint32_t *flags) {
  const size_t i0 = (size_t)blockIdx.x * (256 * CHECK_PER) + threadIdx.x;
  K k[CHECK_PER], prev[CHECK_PER];
#pragma unroll
  for (int j = 0; j < CHECK_PER; j++) {
    const size_t i = i0 + 256 * j;
    if (i < nn) {
      k[j] = nodes[i];
      prev[j] = nodes[i > 0 ? i - 1 : 0];
    }
  }
  bool ok = true;
#pragma unroll
  for (int j = 0; j < CHECK_PER; j++) {
    const size_t i = i0 + 256 * j;
    if (i < nn) ok = ok && node_follows(i > 0, node_wide(prev[j]), node_wide(k[j]), Lm);
  }
  if (!ok) set_flag(flags, DGF_INTERNAL);
}

// the sorted nodes of the balanced refinement; d_hist: per level the nodes (an
// input that has them) or the leaves' parents with repeats, `room` their sum
template <typename K>
static size_t balance_nodes(Context &ctx, const Octree &in, unsigned top, const unsigned long long *d_hist, size_t room,
                            bool inc_corner, DBuf<K> &a, DBuf<K> &b, K **sorted) {
  cudaStream_t s = ctx.stream;
  const unsigned D = in.max_depth, Lm = top - 1;
  ensure_smem_attr(ctx, k_bal_level<K>, (int)sizeof(BalSmem<K>));
  int per_sm = 1;
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bal_level<K>, BAL_TILE, sizeof(BalSmem<K>)));
  DBuf<BalCounts> counts(1, s);
  BalCounts *cnt = counts.get();
  BalCounts h;
  DBuf<K> start(room, s), grown;
  // balanced octrees of the workloads' clouds have 1.3 to 1.9 times the nodes
  // of their input: room for 3 times, and four times that on each retry
  for (size_t grow = 2;; grow *= 4) {
    const size_t cap = grow * room + 65536;
    size_t slots = 1024;
    while (slots < room + cap) slots <<= 1;
    grown.alloc(cap, s);
    DBuf<K> tab(slots, s);
    DG_CUDA(cudaMemsetAsync(tab.get(), 0xff, slots * sizeof(K), s));
    DG_CUDA(cudaMemsetAsync(cnt, 0, sizeof(BalCounts), s));
    DG_CUDA(cudaMemcpyAsync(cnt->room, d_hist, sizeof(cnt->room), cudaMemcpyDeviceToDevice, s));
    {
      ProfScope _prof(ctx, "bal_start", in.nodes ? (double)room * 3 * sizeof(K)
                                                 : (double)in.n * 16 + (double)room * 2 * sizeof(K));
      if (in.nodes)
        k_bal_start<K, false><<<grid_for(in.n_node, 256), 256, 0, s>>>(in.nodes, in.n_node, D, Lm, tab.get(),
                                                                       slots - 1, start.get(), room, cnt, ctx.d_flags);
      else
        k_bal_start<K, true><<<grid_for(in.n, 256), 256, 0, s>>>(in.keys, in.n, D, Lm, tab.get(), slots - 1,
                                                                 start.get(), room, cnt, ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    const unsigned grid =
        grid_for(room + cap, BAL_TILE, (unsigned)(std::max(per_sm, 1) * ctx.num_sms));
    for (unsigned l = Lm; l >= 1; l--) {
      ProfScope _prof(ctx, "bal_level", 0.0);
      k_bal_level<K><<<grid, BAL_TILE, sizeof(BalSmem<K>), s>>>(l, Lm, inc_corner, tab.get(), slots - 1, start.get(),
                                                                grown.get(), cap, cnt, ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    static_assert(sizeof(BalCounts) <= 96 * sizeof(unsigned long long), "the counts fit the pinned mirror");
    DG_CUDA(cudaMemcpyAsync(ctx.h_scratch, cnt, sizeof(BalCounts), cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));
    std::memcpy(&h, ctx.h_scratch, sizeof(h));
    const uint32_t f = read_scalar(ctx, ctx.d_flags);
    if (!(f & DGF_CAPACITY)) break;
    DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
    if (cap > ((size_t)1 << 40) / sizeof(K)) fail(DG_ERR_OUT_OF_MEMORY, "balanceOctree: too many octants");
  }
  BalGather g;
  size_t off = 0, n0 = 0, n1 = 0;
  for (int l = 0; l < 32; l++) {
    g.off[l] = off;
    g.num[l] = h.start[l];
    g.to[l] = n0;
    off += h.room[l];
    n0 += h.start[l];
    n1 += h.grown[l];
  }
  const size_t nn = n0 + n1;
  a.alloc(nn, s);
  b.alloc(nn, s);
  {
    ProfScope _prof(ctx, "bal_gather", (double)nn * 2 * sizeof(K));
    k_bal_gather<K><<<grid_for(room, 256), 256, 0, s>>>(start.get(), g, room, a.get());
    DG_LAUNCH_CHECK();
  }
  if (n1) DG_CUDA(cudaMemcpyAsync(a.get() + n0, grown.get(), n1 * sizeof(K), cudaMemcpyDeviceToDevice, s));
  *sorted = radix_sort<K>(ctx, a.get(), b.get(), nn, 3 * (int)Lm + 5 + (int)in.seg_bits);
  {
    ProfScope _prof(ctx, "bal_check", (double)nn * sizeof(K));
    k_bal_check<K><<<grid_for(nn, 256 * CHECK_PER), 256, 0, s>>>(*sorted, nn, Lm, ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  return nn;
}

void balance_octree(Context &ctx, const Octree &in, Octree &out, bool inc_corner) {
  cudaStream_t s = ctx.stream;
  const unsigned D = in.max_depth;
  const size_t nseg = in.nseg;
  out.max_depth = D;
  out.nseg = nseg;
  out.seg_bits = in.seg_bits;
  const size_t n = in.n;
  if (n == 0) fail(DG_ERR_INVALID_ARG, "balanceOctree: empty input");
  unsigned long long *d_hist = ctx.d_scratch + 16;
  DG_CUDA(cudaMemsetAsync(d_hist, 0, 32 * sizeof(unsigned long long), s));
  DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
  unsigned top = in.top;  // deepest leaf level
  size_t room = in.n_node;
  if (in.nodes) {
    ProfScope _prof(ctx, "bal_node_levels", (double)in.n_node * (in.node_wide ? 16 : 8));
    const unsigned g = grid_for(in.n_node, 256, ctx.num_sms * 8);
    if (in.node_wide)
      k_bal_node_levels<Key128><<<g, 256, 0, s>>>(static_cast<const Key128 *>(in.nodes), in.n_node, d_hist);
    else
      k_bal_node_levels<uint64_t><<<g, 256, 0, s>>>(static_cast<const uint64_t *>(in.nodes), in.n_node, d_hist);
    DG_LAUNCH_CHECK();
  } else {
    // parents per level + domain validation
    {
      ProfScope _prof(ctx, "bal_scan", (double)n * 16);
      k_bal_scan<<<grid_for(n, 256, ctx.num_sms * 8), 256, 0, s>>>(in.keys, n, D, nseg, d_hist, ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 16, d_hist, 32 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    check_device_flags(ctx, "balanceOctree (octant outside the domain or misaligned)");
    top = 0;
    for (unsigned l = 0; l < 32; l++) {
      room += ctx.h_scratch[16 + l];
      if (ctx.h_scratch[16 + l]) top = l + 1;
    }
  }
  DBuf<Key128> res;
  DBuf<uint64_t> seg_off;
  size_t nn = 0;
  auto run = [&](auto tag) {
    typedef decltype(tag) K;
    DBuf<K> a, b;
    K *nodes = nullptr;
    if (room) nn = balance_nodes<K>(ctx, in, top, d_hist, room, inc_corner, a, b, &nodes);
    emit_octree<K>(ctx, nodes, nn, top ? top - 1 : 0, D, nseg, res, seg_off);
    check_device_flags(ctx, "balanceOctree");
    if (nn) keep_nodes(out, nodes == a.get() ? a : b, nn, top);
  };
  if (in.nodes ? !in.node_wide : top == 0 || nodes_fit_64(top, in.seg_bits)) run(uint64_t());
  else run(Key128());
  out.n = 7 * nn + nseg;
  out.keys = res.release_ptr();
  out.seg_off = nseg > 1 ? seg_off.release_ptr() : nullptr;
}

// ------------------------------------------------------------------------
// coarsenOctree (src/coarsen.cpp:53): every complete family of 8 sibling
// leaves is replaced by its parent.  On a sorted, linear, complete octree
// the reference's rule (a first child followed by 7 octants that are not
// first children) is exactly "the 8 octants from a first child are the 8
// children of one parent"; a batch never merges across clouds because the
// parent test includes the cloud bits.
// ------------------------------------------------------------------------
__device__ __forceinline__ unsigned key_child(Key128 k, unsigned D) {
  unsigned l = tag_level(k);
  if (l == 0) return 0;
  return (unsigned)(key_shr(tag_anchor(k), 3 * (D - l)).lo & 7u);
}
__device__ __forceinline__ Key128 key_parent(Key128 k, unsigned D) {
  unsigned l = tag_level(k);
  unsigned sh = 3 * (D - l + 1);
  return make_tagged(key_shl(key_shr(tag_anchor(k), sh), sh), l - 1);
}

__global__ void k_coarsen_mark(const Key128 *__restrict__ k, size_t n, unsigned D, uint32_t *__restrict__ fam) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Key128 ki = k[i];
  const unsigned l = tag_level(ki);
  bool start = l >= 1 && key_child(ki, D) == 0 && i + 7 < n;
  if (start) {
    const Key128 par = key_parent(ki, D);
    for (int j = 1; j < 8 && start; j++) {
      Key128 kj = k[i + j];
      start = tag_level(kj) == l && key_eq(key_parent(kj, D), par);
    }
  }
  fam[i] = start ? 1u : 0u;
}

__global__ void k_coarsen_apply(const Key128 *__restrict__ k, size_t n, unsigned D, const uint32_t *__restrict__ fam,
                                Key128 *__restrict__ val, uint32_t *__restrict__ keep) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Key128 ki = k[i];
  const unsigned c = key_child(ki, D);
  const bool member = c >= 1 && i >= c && fam[i - c];
  keep[i] = member ? 0u : 1u;
  val[i] = fam[i] ? key_parent(ki, D) : ki;
}

// the nodes that stay: those with a node among their children, which follows
// them in preorder
template <typename K>
__global__ void k_coarsen_flags(const K *__restrict__ nodes, size_t nn, unsigned Lm, uint32_t *__restrict__ keep) {
  typedef typename NodeWide<K>::W W;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const W k = node_wide(nodes[i]);
  const unsigned d = (unsigned)k & 31u;
  keep[i] = i + 1 < nn && (node_wide(nodes[i + 1]) >> 5) < (k >> 5) + ((W)1 << (3 * (Lm - d))) ? 1u : 0u;
}
// ... with paths to one level less (the deepest nodes have no node below)
template <typename K>
__global__ void k_coarsen_nodes(const K *__restrict__ nodes, const uint32_t *__restrict__ keep,
                                const uint32_t *__restrict__ pos, size_t nn, K *__restrict__ out) {
  typedef NodeWide<K> N;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn || !keep[i]) return;
  const typename N::W k = node_wide(nodes[i]);
  out[pos[i]] = N::narrow(k >> 8 << 5 | (k & 31u));
}

template <typename K>
static void coarsen_nodes(Context &ctx, const Octree &in, Octree &out, bool leaves) {
  cudaStream_t s = ctx.stream;
  const K *nodes = static_cast<const K *>(in.nodes);
  const size_t nn = in.n_node;
  DBuf<uint32_t> keep(nn, s), pos(nn, s);
  uint32_t *d_total = reinterpret_cast<uint32_t *>(ctx.d_scratch);
  {
    ProfScope _prof(ctx, "coarsen_flags", (double)nn * (sizeof(K) + 4));
    k_coarsen_flags<K><<<grid_for(nn, 256), 256, 0, s>>>(nodes, nn, in.top - 1, keep.get());
    DG_LAUNCH_CHECK();
  }
  exclusive_scan<uint32_t, uint32_t>(keep.get(), pos.get(), nn, d_total, s);
  const size_t nc = read_scalar(ctx, d_total);
  DBuf<K> kept(nc ? nc : 1, s);
  DBuf<Key128> res;
  DBuf<uint64_t> seg_off;
  if (nc) {
    ProfScope _prof(ctx, "coarsen_nodes", (double)nn * 8 + (double)nc * 2 * sizeof(K));
    k_coarsen_nodes<K><<<grid_for(nn, 256), 256, 0, s>>>(nodes, keep.get(), pos.get(), nn, kept.get());
    DG_LAUNCH_CHECK();
  }
  if (leaves || !nc)
    emit_octree<K>(ctx, kept.get(), nc, nc ? in.top - 2 : 0, in.max_depth, 1, res, seg_off);
  out.n = 7 * nc + 1;
  out.keys = res.release_ptr();
  if (nc) keep_nodes(out, kept, nc, in.top - 1);
}

void coarsen_octree(Context &ctx, const Octree &in, Octree &out, bool leaves) {
  cudaStream_t s = ctx.stream;
  const size_t n = in.n;
  out = Octree();
  out.max_depth = in.max_depth;
  out.nseg = in.nseg;
  out.seg_bits = in.seg_bits;
  if (in.nseg != 1) fail(DG_ERR_UNSUPPORTED, "coarsenOctree: one cloud per call");
  if (in.nodes) {
    if (in.node_wide) coarsen_nodes<Key128>(ctx, in, out, leaves);
    else coarsen_nodes<uint64_t>(ctx, in, out, leaves);
    return;
  }
  DBuf<Key128> res(n ? n : 1, s);
  if (n < 8) {  // coarsen.cpp:66-70
    if (n) DG_CUDA(cudaMemcpyAsync(res.get(), in.keys, n * sizeof(Key128), cudaMemcpyDeviceToDevice, s));
    DG_CUDA(cudaStreamSynchronize(s));
    out.n = n;
    out.keys = res.release_ptr();
    return;
  }
  DBuf<uint32_t> fam(n, s), keep(n, s);
  DBuf<Key128> val(n, s);
  {
    ProfScope _prof(ctx, "coarsen_mark", (double)n * 20);
    k_coarsen_mark<<<grid_for(n, 256), 256, 0, s>>>(in.keys, n, in.max_depth, fam.get());
    DG_LAUNCH_CHECK();
  }
  {
    ProfScope _prof(ctx, "coarsen_apply", (double)n * 40);
    k_coarsen_apply<<<grid_for(n, 256), 256, 0, s>>>(in.keys, n, in.max_depth, fam.get(), val.get(), keep.get());
    DG_LAUNCH_CHECK();
  }
  out.n = compact<Key128>(ctx, val.get(), keep.get(), n, res.get());
  out.keys = res.release_ptr();
}

// ------------------------------------------------------------------------
// completeOctree (src/construct.cpp:518).  At one rank the reference runs its
// general path (:534-700): the tree sort's sort + duplicate + ancestor
// removal when the input is not declared unique (include/sfcSort.h:532-575),
// a plain sort when it is unique but not declared sorted, then
// appendCompleteRegion (:1077) between consecutive octants, an octant that is
// followed by its own descendant being left out.  The filled gaps are the
// maximal aligned Morton blocks between consecutive leaves (the same blocks
// appendCompleteRegion emits), so the construction's gap kernels apply.
// ------------------------------------------------------------------------
// sort form: the Morton anchor above the 5 level bits, so that a radix sort
// over the low 3D + 5 bits gives the reference's order (on equal anchors the
// coarser octant first)
__global__ void k_to_sortform(const Key128 *__restrict__ in, size_t n, Key128 *__restrict__ out) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = key_or(key_shl(tag_anchor(in[i]), 5), Key128{(uint64_t)tag_level(in[i]), 0});
}

__global__ void k_from_sortform(const Key128 *__restrict__ in, size_t n, Key128 *__restrict__ out) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_tagged(key_shr(in[i], 5), (unsigned)(in[i].lo & 31u));
}

// octant i is kept unless its successor is its descendant; an order that
// breaks the caller's declaration raises DGF_ORDER
__global__ void k_complete_leaves(const Key128 *__restrict__ s, size_t n, unsigned D, bool strict,
                                  Key128 *__restrict__ val, uint32_t *__restrict__ keep, uint32_t *flags) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Key128 a = s[i];
  const unsigned la = (unsigned)(a.lo & 31u);
  bool k = true;
  if (i + 1 < n) {
    const Key128 b = s[i + 1];
    if (key_lt(b, a) || (strict && key_eq(a, b))) atomicOr(flags, DGF_ORDER);
    const unsigned lb = (unsigned)(b.lo & 31u);
    if (la < lb) {
      const unsigned sh = 5 + 3 * (D - la);
      k = !key_eq(key_shr(a, sh), key_shr(b, sh));
    }
  }
  val[i] = make_tagged(key_shr(a, 5), la);
  keep[i] = k ? 1u : 0u;
}

// ------------------------------------------------------------------------
// one cloud of a batch as its own octree (cloud bits cleared)
// ------------------------------------------------------------------------
__global__ void k_strip_cloud(const Key128 *__restrict__ in, size_t n, unsigned D, Key128 *__restrict__ out) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_tagged(morton_part(in[i], D), tag_level(in[i]));
}

template <typename K>
__global__ void k_strip_nodes(const K *__restrict__ in, size_t n, unsigned Lm, K *__restrict__ out) {
  typedef NodeWide<K> N;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = N::narrow(node_wide(in[i]) & (((typename N::W)1 << (3 * Lm + 5)) - 1));
}

void octree_extract(Context &ctx, const Octree &in, size_t seg, Octree &out) {
  if (seg >= in.nseg) fail(DG_ERR_INVALID_ARG, "octree: cloud index out of range");
  uint64_t off[2] = {0, in.n};
  if (in.nseg > 1)
    DG_CUDA(cudaMemcpyAsync(off, in.seg_off + seg, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx.stream));
  DG_CUDA(cudaStreamSynchronize(ctx.stream));
  const size_t n = off[1] - off[0];
  out = Octree();
  out.max_depth = in.max_depth;
  out.n = n;
  DBuf<Key128> k(n ? n : 1, ctx.stream);
  if (n) {
    ProfScope _prof(ctx, "strip_cloud", (double)n * 32);
    k_strip_cloud<<<grid_for(n, 256), 256, 0, ctx.stream>>>(in.keys + off[0], n, in.max_depth, k.get());
    DG_LAUNCH_CHECK();
  }
  // the cloud's nodes: 7 leaves per node and one more per cloud lie before them
  const size_t first = (off[0] - seg) / 7, nn = n ? (n - 1) / 7 : 0;
  auto strip = [&](auto tag) {
    typedef decltype(tag) K;
    DBuf<K> nodes(nn, ctx.stream);
    k_strip_nodes<K><<<grid_for(nn, 256), 256, 0, ctx.stream>>>(static_cast<const K *>(in.nodes) + first, nn,
                                                                in.top - 1, nodes.get());
    DG_LAUNCH_CHECK();
    keep_nodes(out, nodes, nn, in.top);
  };
  if (in.nodes && nn) {
    if (in.node_wide) strip(Key128());
    else strip(uint64_t());
  }
  out.keys = k.release_ptr();
}

// ------------------------------------------------------------------------
// conversions
// ------------------------------------------------------------------------
// (a single cloud may hold octants just outside its domain: the reference's
// construction emits them for some inputs with repeated points; their
// anchor bits then run past 3D and are decoded as is)
// Four records per thread, their keys loaded together: with one the loads in
// flight and the operations of demorton3 (in 64-bit pieces) took 0.67 ms for
// 8.8e7 records, with one and 32-bit pieces 0.57, now 0.51 ms (5.5 TB/s).
constexpr int XYZL_PER = 4;
__global__ void __launch_bounds__(256) k_to_xyzl(const Key128 *__restrict__ k, size_t n, unsigned D, bool batched,
                                                 uint4 *__restrict__ out) {
  const size_t i0 = (size_t)blockIdx.x * (256 * XYZL_PER) + threadIdx.x;
  Key128 key[XYZL_PER];
#pragma unroll
  for (int j = 0; j < XYZL_PER; j++)
    if (i0 + 256 * j < n) key[j] = k[i0 + 256 * j];
#pragma unroll
  for (int j = 0; j < XYZL_PER; j++) {
    if (i0 + 256 * j >= n) break;
    uint32_t x, y, z;
    demorton3(batched ? morton_part(key[j], D) : tag_anchor(key[j]), x, y, z);
    out[i0 + 256 * j] = make_uint4(x, y, z, tag_level(key[j]));
  }
}

__global__ void k_from_xyzl(const uint4 *__restrict__ in, size_t n, unsigned D, Key128 *__restrict__ out,
                            uint32_t *flags) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint4 v = in[i];
  unsigned lev = v.w & 31u;
  uint64_t len = 1ull << (D - min(lev, D));
  uint64_t dom = 1ull << D;
  bool ok = lev <= D && v.x % len == 0 && v.y % len == 0 && v.z % len == 0 && v.x < dom && v.y < dom && v.z < dom;
  if (!ok) atomicOr(flags, DGF_DOMAIN);
  out[i] = make_tagged(morton3(v.x, v.y, v.z), lev);
}

// ------------------------------------------------------------------------
// Hilbert order (the reference's default build, -DHILBERT_ORDERING:
// TreeNode::operator< include/TreeNode.tcc:130-210 with the tables of
// src/hcurvedata.cpp:329-520).  The curve is self-similar: a cell's 8
// children are visited in the order HIL_BASE_ORDER, transformed by the
// cell's own symmetry, and each child's cell carries its parent's symmetry
// composed with HIL_CHILD_SYM of its base position.  A state table of the
// reachable symmetries (24) is generated from these two rows; an octant's
// key is its child ranks root to leaf (3 bits per level), padded to maxDepth,
// above its level, which orders octants as the reference's comparison does
// (an ancestor before its descendants).
// ------------------------------------------------------------------------
namespace {
// corner index c = x | y << 1 | z << 2
constexpr uint8_t HIL_BASE_ORDER[8] = {0, 2, 3, 1, 5, 7, 6, 4};
// child symmetry per base corner: new bit i = old bit perm[i] ^ bit i of flip
struct CubeSym {
  uint8_t perm[3];
  uint8_t flip;
};
constexpr CubeSym HIL_CHILD_SYM[8] = {{{0, 2, 1}, 0}, {{2, 0, 1}, 6}, {{2, 1, 0}, 0}, {{0, 1, 2}, 0},
                                      {{0, 2, 1}, 6}, {{2, 0, 1}, 3}, {{2, 1, 0}, 5}, {{0, 1, 2}, 0}};
constexpr int HIL_MAX_STATES = 32;

struct HilbertTable {
  uint8_t e[HIL_MAX_STATES * 8];  // [state][corner]: rank | next state << 3
};

HilbertTable build_hilbert_table() {
  using Map = std::array<uint8_t, 8>;  // a symmetry as its action on corners
  auto sym_map = [](const CubeSym &g) {
    Map m{};
    for (unsigned c = 0; c < 8; c++) {
      unsigned r = 0;
      for (unsigned i = 0; i < 3; i++) r |= (((c >> g.perm[i]) & 1u) ^ ((g.flip >> i) & 1u)) << i;
      m[c] = (uint8_t)r;
    }
    return m;
  };
  uint8_t rank0[8];
  for (unsigned k = 0; k < 8; k++) rank0[HIL_BASE_ORDER[k]] = (uint8_t)k;
  std::vector<Map> states;
  Map id{};
  for (unsigned c = 0; c < 8; c++) id[c] = (uint8_t)c;
  states.push_back(id);
  HilbertTable t{};
  for (size_t s = 0; s < states.size(); s++) {
    const Map g = states[s];
    Map ginv{};
    for (unsigned c = 0; c < 8; c++) ginv[g[c]] = (uint8_t)c;
    for (unsigned c = 0; c < 8; c++) {
      const unsigned c0 = ginv[c];
      const Map tc = sym_map(HIL_CHILD_SYM[c0]);
      Map child{};
      for (unsigned q = 0; q < 8; q++) child[q] = g[tc[q]];
      size_t id2 = std::find(states.begin(), states.end(), child) - states.begin();
      if (id2 == states.size()) {
        if (states.size() == HIL_MAX_STATES) fail(DG_ERR_INTERNAL, "Hilbert table: too many states");
        states.push_back(child);
      }
      t.e[s * 8 + c] = (uint8_t)(rank0[c0] | (id2 << 3));
    }
  }
  return t;
}

const HilbertTable &hilbert_table() {
  static const HilbertTable t = build_hilbert_table();
  return t;
}
}  // namespace

// key[i] = (Hilbert rank path << 5 | level) << 32 | i for the octants of
// one cloud (i < 2^32)
__global__ void k_hilbert_keys(const Key128 *__restrict__ k, size_t n, unsigned D, bool batched, HilbertTable tab,
                               Key128 *__restrict__ out) {
  __shared__ uint8_t t[HIL_MAX_STATES * 8];
  for (int i = threadIdx.x; i < HIL_MAX_STATES * 8; i += blockDim.x) t[i] = tab.e[i];
  __syncthreads();
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t x, y, z;
  demorton3(batched ? morton_part(k[i], D) : tag_anchor(k[i]), x, y, z);
  const unsigned lev = tag_level(k[i]);
  u128 h = 0;
  unsigned st = 0;
  for (unsigned l = 0; l < lev; l++) {
    const unsigned b = D - 1 - l;
    const unsigned c = ((x >> b) & 1u) | (((y >> b) & 1u) << 1) | (((z >> b) & 1u) << 2);
    const unsigned e = t[st * 8 + c];
    h = (h << 3) | (e & 7u);
    st = e >> 3;
  }
  h <<= 3 * (D - lev);
  out[i] = from_u128((((h << 5) | lev) << 32) | (u128)(uint32_t)i);
}

__global__ void k_gather_xyzl(const Key128 *__restrict__ k, const Key128 *__restrict__ order, size_t n, unsigned D,
                              bool batched, uint4 *__restrict__ out) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Key128 v = k[(uint32_t)order[i].lo];
  uint32_t x, y, z;
  demorton3(batched ? morton_part(v, D) : tag_anchor(v), x, y, z);
  out[i] = make_uint4(x, y, z, tag_level(v));
}

// records of o in Hilbert order, cloud by cloud
static void octree_to_xyzl_hilbert(Context &ctx, const Octree &o, uint32_t *d_xyzl) {
  cudaStream_t s = ctx.stream;
  const unsigned D = o.max_depth;
  std::vector<uint64_t> off{0, (uint64_t)o.n};
  if (o.nseg > 1) {
    off.resize(o.nseg + 1);
    DG_CUDA(cudaMemcpyAsync(off.data(), o.seg_off, (o.nseg + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    DG_CUDA(cudaStreamSynchronize(s));
  }
  const HilbertTable &tab = hilbert_table();
  DBuf<Key128> a(o.n, s), b(o.n, s);
  for (size_t g = 0; g + 1 < off.size(); g++) {
    const size_t n = off[g + 1] - off[g];
    if (!n) continue;
    if (n > 0xffffffffull) fail(DG_ERR_UNSUPPORTED, "Hilbert order: more than 2^32 octants in one cloud");
    ProfScope _prof(ctx, "hilbert_order", (double)n * 16 * 36);
    k_hilbert_keys<<<grid_for(n, 256), 256, 0, s>>>(o.keys + off[g], n, D, o.nseg > 1, tab, a.get() + off[g]);
    DG_LAUNCH_CHECK();
    Key128 *srt = radix_sort<Key128>(ctx, a.get() + off[g], b.get() + off[g], n, 3 * (int)D + 5 + 32, 0, true);
    check_device_flags(ctx, "Hilbert order");
    k_gather_xyzl<<<grid_for(n, 256), 256, 0, s>>>(o.keys + off[g], srt, n, D, o.nseg > 1,
                                                   reinterpret_cast<uint4 *>(d_xyzl) + off[g]);
    DG_LAUNCH_CHECK();
  }
}

void octree_to_xyzl(Context &ctx, const Octree &o, uint32_t *d_xyzl) {
  if (!o.n) return;
  if (ctx.order == 1) {
    octree_to_xyzl_hilbert(ctx, o, d_xyzl);
    return;
  }
  {
    ProfScope _prof("to_xyzl", (double)o.n * 32);
    k_to_xyzl<<<grid_for(o.n, 256 * XYZL_PER), 256, 0, ctx.stream>>>(o.keys, o.n, o.max_depth, o.nseg > 1,
                                                          reinterpret_cast<uint4 *>(d_xyzl));
    DG_LAUNCH_CHECK();
  }
}

void octree_from_xyzl(Context &ctx, const uint32_t *d_xyzl, size_t n, unsigned D, Octree &out) {
  out.max_depth = D;
  out.n = n;
  DBuf<Key128> k(n, ctx.stream);
  if (n) {
    {
      ProfScope _prof("from_xyzl", (double)n * 32);
      k_from_xyzl<<<grid_for(n, 256), 256, 0, ctx.stream>>>(reinterpret_cast<const uint4 *>(d_xyzl), n, D, k.get(),
                                                            ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    check_device_flags(ctx, "octree upload");
    if (ctx.order == 1) {  // records in Hilbert order: the device keeps Morton order
      DBuf<Key128> a(n, ctx.stream), b(n, ctx.stream);
      k_to_sortform<<<grid_for(n, 256), 256, 0, ctx.stream>>>(k.get(), n, a.get());
      DG_LAUNCH_CHECK();
      Key128 *srt = radix_sort<Key128>(ctx, a.get(), b.get(), n, 3 * (int)D + 5, 0, true);
      check_device_flags(ctx, "Hilbert order");
      k_from_sortform<<<grid_for(n, 256), 256, 0, ctx.stream>>>(srt, n, k.get());
      DG_LAUNCH_CHECK();
    }
  }
  out.keys = k.release_ptr();
}

void octree_free(Context &ctx, Octree &o) {
  if (o.keys) cudaFreeAsync(o.keys, ctx.stream);
  if (o.seg_off) cudaFreeAsync(o.seg_off, ctx.stream);
  if (o.nodes) cudaFreeAsync(o.nodes, ctx.stream);
  o = Octree();
}

void complete_octree(Context &ctx, const uint32_t *d_xyzl, size_t n, unsigned D, bool is_unique, bool is_sorted,
                     Octree &out) {
  cudaStream_t s = ctx.stream;
  out = Octree();
  out.max_depth = D;
  if (n == 0) return;  // construct.cpp:587: nothing to complete
  DBuf<Key128> a(n, s), b(n, s);
  {
    ProfScope _prof(ctx, "complete_sortform", (double)n * 48);
    k_from_xyzl<<<grid_for(n, 256), 256, 0, s>>>(reinterpret_cast<const uint4 *>(d_xyzl), n, D, b.get(),
                                                 ctx.d_flags);
    DG_LAUNCH_CHECK();
    k_to_sortform<<<grid_for(n, 256), 256, 0, s>>>(b.get(), n, a.get());
    DG_LAUNCH_CHECK();
  }
  check_device_flags(ctx, "completeOctree");  // domain and alignment of the records
  const int bits = 3 * (int)D + 5;
  if (ctx.order == 1) is_sorted = false;  // records in Hilbert order: sorted into Morton order here
  Key128 *sorted = a.get();
  size_t m = n;
  if (!is_unique) m = sort_unique<Key128>(ctx, a.get(), b.get(), n, bits, &sorted);
  else if (!is_sorted) sorted = radix_sort<Key128>(ctx, a.get(), b.get(), n, bits, 0, true);
  Key128 *other = (sorted == a.get()) ? b.get() : a.get();
  DBuf<uint32_t> keep(m, s);
  {
    ProfScope _prof(ctx, "complete_leaves", (double)m * 36);
    k_complete_leaves<<<grid_for(m, 256), 256, 0, s>>>(sorted, m, D, is_unique, other, keep.get(), ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  check_device_flags(ctx, "completeOctree");
  const size_t ns = compact<Key128>(ctx, other, keep.get(), m, sorted);
  keep.release();
  const u128 total = (u128)1 << (3 * D);
  DBuf<uint32_t> cnt(ns, s);
  {
    ProfScope _prof(ctx, "fill_count", (double)ns * 20);
    k_fill_count<<<grid_for(ns, 256), 256, 0, s>>>(sorted, ns, D, total, cnt.get());
    DG_LAUNCH_CHECK();
  }
  DBuf<uint64_t> off(ns, s);
  uint64_t *d_total = reinterpret_cast<uint64_t *>(ctx.d_scratch);
  exclusive_scan<uint32_t, uint64_t>(cnt.get(), off.get(), ns, d_total, s);
  const size_t nout = (size_t)read_scalar(ctx, d_total);
  DBuf<Key128> res(nout, s);
  {
    ProfScope _prof(ctx, "fill_emit", (double)ns * 24);
    k_fill_emit<<<grid_for(ns, 256), 256, 0, s>>>(sorted, ns, D, total, off.get(), res.get());
    DG_LAUNCH_CHECK();
  }
  out.n = nout;
  out.keys = res.release_ptr();
}

// par::sampleSort (include/parUtils.h:424; at one rank a local sort,
// src/parUtils.tcc:1868-1875) and par::removeDuplicates (parUtils.h:437) of
// octant records: sorted in the octant order (ancestor first on equal
// anchors), repeated records removed when asked (mode 1).  Mode 2 is the
// TS_REMOVE_DUPLICATES output of SFC::seqSort::SFC_treeSort
// (include/sfcSort.h:532-575): sorted, repeated records removed, and every
// octant followed by one of its descendants removed (the descendants of an
// octant follow it contiguously in any space-filling-curve order).
void sort_octants(Context &ctx, const uint32_t *d_xyzl, size_t n, unsigned D, int mode, Octree &out) {
  const bool unique = mode != 0;
  cudaStream_t s = ctx.stream;
  out = Octree();
  out.max_depth = D;
  if (n == 0) return;
  DBuf<Key128> a(n, s), b(n, s);
  {
    ProfScope _prof(ctx, "sort_octants_keys", (double)n * 48);
    k_from_xyzl<<<grid_for(n, 256), 256, 0, s>>>(reinterpret_cast<const uint4 *>(d_xyzl), n, D, b.get(),
                                                 ctx.d_flags);
    DG_LAUNCH_CHECK();
    k_to_sortform<<<grid_for(n, 256), 256, 0, s>>>(b.get(), n, a.get());
    DG_LAUNCH_CHECK();
  }
  check_device_flags(ctx, "sortOctants");
  const int bits = 3 * (int)D + 5;
  Key128 *srt = a.get();
  size_t m = n;
  if (unique) m = sort_unique<Key128>(ctx, a.get(), b.get(), n, bits, &srt);
  else {
    srt = radix_sort<Key128>(ctx, a.get(), b.get(), n, bits, 0, true);
    check_device_flags(ctx, "sortOctants");
  }
  if (mode == 2) {
    // tagged keys of the octants not followed by a descendant
    Key128 *other = (srt == a.get()) ? b.get() : a.get();
    DBuf<uint32_t> keep(m, s);
    {
      ProfScope _prof(ctx, "treesort_leaves", (double)m * 36);
      k_complete_leaves<<<grid_for(m, 256), 256, 0, s>>>(srt, m, D, true, other, keep.get(), ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    DBuf<Key128> res(m, s);
    const size_t nk = compact<Key128>(ctx, other, keep.get(), m, res.get());
    check_device_flags(ctx, "SFC_treeSort");
    out.n = nk;
    out.keys = res.release_ptr();
    return;
  }
  DBuf<Key128> res(m, s);
  k_from_sortform<<<grid_for(m, 256), 256, 0, s>>>(srt, m, res.get());
  DG_LAUNCH_CHECK();
  out.n = m;
  out.keys = res.release_ptr();
}

// ------------------------------------------------------------------------
namespace {
__global__ void k_selftest_keys(uint64_t *k, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) k[i] = (i * 0x9E3779B97F4A7C15ull) >> 7;  // every low digit occurs
}
}  // namespace

void lookback_timeout_selftest(Context &ctx, size_t n, unsigned skipped) {
  using K = uint64_t;
  constexpr size_t TILE = (size_t)RS_BLOCK * OsCfg<K>::ITEMS;
  const size_t ntiles = (n + TILE - 1) / TILE;
  if (skipped == 0 || ntiles <= skipped || ntiles > (1u << 20))
    fail(DG_ERR_INVALID_ARG, "look-back self-test: need 1 <= skipped < tiles <= 2^20");
  cudaStream_t s = ctx.stream;
  DBuf<K> in(n, s), out(n, s);
  DBuf<uint64_t> status(ntiles * 256, s), doffs(256, s);
  k_selftest_keys<<<grid_for(n, 256), 256, 0, s>>>(in.get(), n);
  DG_LAUNCH_CHECK();
  // digit offsets of the low byte (exclusive scan of its histogram), so
  // every write of the pass stays inside [0, n)
  std::vector<uint64_t> h(256, 0), offs(256, 0);
  std::vector<K> keys(n);
  DG_CUDA(cudaMemcpyAsync(keys.data(), in.get(), n * sizeof(K), cudaMemcpyDeviceToHost, s));
  DG_CUDA(cudaStreamSynchronize(s));
  for (K k : keys) h[k & 255]++;
  for (int d = 1; d < 256; d++) offs[d] = offs[d - 1] + h[d - 1];
  DG_CUDA(cudaMemcpyAsync(doffs.get(), offs.data(), 256 * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  DG_CUDA(cudaMemsetAsync(status.get(), 0, ntiles * 256 * sizeof(uint64_t), s));
  // the tile tickets start at `skipped`: tiles [0, skipped) are never
  // processed and their status words stay unpublished
  unsigned *d_counter = reinterpret_cast<unsigned *>(ctx.d_scratch + 12);
  const unsigned start = skipped;
  DG_CUDA(cudaMemcpyAsync(d_counter, &start, sizeof(unsigned), cudaMemcpyHostToDevice, s));
  k_rs_onesweep<K, OsCfg<K>::ITEMS><<<(unsigned)(ntiles - skipped), RS_BLOCK, 0, s>>>(
      in.get(), out.get(), n, 0, doffs.get(), status.get(), d_counter, ctx.d_flags);
  DG_LAUNCH_CHECK();
  check_device_flags(ctx, "look-back self-test");
}

}  // namespace dg
