// Octree mesh build (ot::DA at one rank: src/oda/oda.cpp:250 ->
// DA_FactoryPart1..3, src/oda/private/odaFactory.cpp, odaBuildNlist.cpp)
// and the Laplacian + mass element loop (examples/src/backend/odaJac.C).
//
// Hanging vertices.  Element e at level l is child c of parent P (level
// l-1).  Only the vertices c^r with r in {1,2,4} (midpoints of P's edges
// through corner c) and r in {3,5,6} (centres of P's faces through corner
// c) can hang.  Such a vertex hangs when one of P's same-size neighbours
// that share that face or edge is an unrefined leaf (2:1 balance bounds the
// neighbour to level l-1).  A hanging vertex k refers to P's vertex k, which
// is always a mesh node; the element type (one of 18 per child number,
// include/oda/cnumEtypes.h) selects the stencil that folds the hanging
// interpolation into the element matrix.
//
// Nodes.  Every node is the anchor of exactly one octant of the reference's
// DA octant set (elements plus the positive-boundary pseudo-octants of
// octFunctions.cpp:681-770).  Here element e owns its anchor (when it does
// not hang) and its vertices on the positive domain boundary, so the node
// set is numbered by one scan over elements; the owner of any vertex is the
// leaf that contains it after clamping boundary coordinates inward.
#include "dg_da.cuh"
#include "dg_elem.cuh"
#include "dg_nodes.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

namespace dg {

// ------------------------------------------------------------------------
// element-type and stencil tables (host)
// ------------------------------------------------------------------------
// The 18 hanging configurations in the reference's type order
// (include/oda/odaUtils.tcc:14-120), as vertex sets relative to the child's
// own corner: relative vertex r = 1, 2, 4 are the edge midpoints, 3, 5, 6 the
// face centres.  Bit r of each entry marks relative vertex r as hanging.
static const uint8_t kCanonRel[18] = {0x00, 0x04, 0x02, 0x06, 0x10, 0x14, 0x12, 0x16, 0x0e,
                                      0x1e, 0x54, 0x56, 0x5e, 0x32, 0x36, 0x3e, 0x76, 0x7e};
// Each child number's table is the canonical one with its axes permuted:
// the relative axis bit that canonical x, y, z map to.
static const uint8_t kAxisPerm[8][3] = {{1, 2, 4}, {2, 1, 4}, {2, 1, 4}, {1, 2, 4},
                                        {1, 4, 2}, {2, 4, 1}, {2, 4, 1}, {1, 4, 2}};

void gen_etype_masks(uint8_t masks[8 * 18]) {
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) {
      uint8_t m = 0;
      for (int r = 0; r < 8; r++) {
        if (!(kCanonRel[t] >> r & 1)) continue;
        int pr = ((r & 1) ? kAxisPerm[c][0] : 0) | ((r & 2) ? kAxisPerm[c][1] : 0) | ((r & 4) ? kAxisPerm[c][2] : 0);
        m |= (uint8_t)(1u << (pr ^ c));
      }
      masks[c * 18 + t] = m;
    }
}

// S[c][t] = P^T K P on the reference element [-1,1]^3 with trilinear shape
// functions; K = stiffness (Laplacian) or mass; P maps the 8 referenced
// values to the child's vertex values (a hanging vertex is the average of
// the parent corners spanning its edge or face).
void gen_stencils(double *lap, double *mass) {
  const double m1[2][2] = {{2.0 / 3.0, 1.0 / 3.0}, {1.0 / 3.0, 2.0 / 3.0}};
  const double a1[2][2] = {{0.5, -0.5}, {-0.5, 0.5}};
  double K[8][8], M[8][8];
  for (int i = 0; i < 8; i++)
    for (int j = 0; j < 8; j++) {
      int ix = i & 1, iy = i >> 1 & 1, iz = i >> 2 & 1, jx = j & 1, jy = j >> 1 & 1, jz = j >> 2 & 1;
      K[i][j] = a1[ix][jx] * m1[iy][jy] * m1[iz][jz] + m1[ix][jx] * a1[iy][jy] * m1[iz][jz] +
                m1[ix][jx] * m1[iy][jy] * a1[iz][jz];
      M[i][j] = m1[ix][jx] * m1[iy][jy] * m1[iz][jz];
    }
  uint8_t masks[8 * 18];
  gen_etype_masks(masks);
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) {
      double P[8][8];
      std::memset(P, 0, sizeof(P));
      uint8_t hm = masks[c * 18 + t];
      for (int k = 0; k < 8; k++) {
        if (!(hm >> k & 1)) {
          P[k][k] = 1.0;
          continue;
        }
        int d = k ^ c, cnt = 0;
        for (int s = 0; s < 8; s++) cnt += ((s & d) == s);
        for (int s = 0; s < 8; s++)
          if ((s & d) == s) P[k][c ^ s] += 1.0 / cnt;
      }
      for (int i = 0; i < 8; i++)
        for (int j = 0; j < 8; j++) {
          double sl = 0.0, sm = 0.0;
          for (int a = 0; a < 8; a++)
            for (int b = 0; b < 8; b++) {
              double w = P[a][i] * P[b][j];
              if (w != 0.0) {
                sl += w * K[a][b];
                sm += w * M[a][b];
              }
            }
          size_t o = (((size_t)c * 18 + t) * 8 + i) * 8 + j;
          lap[o] = sl;
          mass[o] = sm;
        }
    }
}


void ensure_stencils(Context &ctx) {
  if (ctx.d_sten64) return;
  std::vector<double> lap(8 * 18 * 64), mass(8 * 18 * 64);
  gen_stencils(lap.data(), mass.data());
  std::vector<double> s64(STEN_ENTRIES);
  for (int ct = 0; ct < 8 * 18; ct++)
    for (int q = 0; q < 64; q++) {
      s64[ct * 128 + q] = lap[ct * 64 + q];
      s64[ct * 128 + 64 + q] = mass[ct * 64 + q];
    }
  uint8_t masks[8 * 18], etype_of[8 * 256];
  gen_etype_masks(masks);
  std::memset(etype_of, 0xff, sizeof(etype_of));
  for (int c = 0; c < 8; c++)
    for (int t = 0; t < 18; t++) etype_of[c * 256 + masks[c * 18 + t]] = (uint8_t)t;
  double *d64 = nullptr;
  uint8_t *det = nullptr;
  DG_CUDA(cudaMalloc((void **)&d64, STEN_ENTRIES * sizeof(double)));
  DG_CUDA(cudaMalloc((void **)&det, sizeof(etype_of)));
  DG_CUDA(cudaMemcpy(d64, s64.data(), STEN_ENTRIES * sizeof(double), cudaMemcpyHostToDevice));
  DG_CUDA(cudaMemcpy(det, etype_of, sizeof(etype_of), cudaMemcpyHostToDevice));
  ctx.d_sten64 = d64;
  ctx.d_etype_of = det;
}

// ------------------------------------------------------------------------
// mesh build
// ------------------------------------------------------------------------
// The build works per family (a node of the octree, dg_nodes.cuh, with its
// children) instead of per element: the elements and lattice of a family are
// found through the nodes around it, of which there are a seventh as many, in
// a table that fits the L2 cache.  Per family that is 7 look-ups of nodes one
// level up, where an element-wise build looks up 6 neighbours and 8 vertices
// for each of 7 elements among all elements.  Mesh of 1e6 points (5.5e6
// elements, 0.79e6 families), all kernels but the element loop's: 1.19 -> 0.74
// ms, of which the look-ups take 0.18 and the lattices 0.26 (loads that depend
// on one another, from L2).  A seventeenth of the nodes have no leaf among
// their children; they are left out of the element loop's families, where each
// would idle a thread (its FP64 form 0.70 -> 0.655 ms).

// the nodes by key: table of keys and the index of each
template <typename K>
__global__ void k_node_table(const K *__restrict__ nodes, size_t nn, unsigned Lm, K *__restrict__ tab,
                             uint32_t *__restrict__ val, uint64_t mask, uint32_t *flags) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn) return;
  const auto key = node_wide(nodes[i]);
  uint64_t h = node_hash(key, Lm) & mask;
  for (int probe = 0; probe < NODE_PROBES; probe++) {
    const auto cur = slot_cas(tab + h, key);
    if (cur == node_empty(key)) {
      val[h] = (uint32_t)i;
      return;
    }
    if (cur == key) {  // twice in the list
      set_flag(flags, DGF_INTERNAL);
      return;
    }
    h = (h + NODE_STEP) & mask;
  }
  set_flag(flags, DGF_CAPACITY);
}

// Per node and child: x the nodes before the child in preorder (its own index
// where it is a node; with KID_LEAF where it is a leaf), y the element anchored
// at the child's anchor (the child itself, or the first leaf below it).  Per
// node which children are leaves, and whether any is.  8 threads per node; the
// search as in the leaf emission (dg_octree.cu): the warp holds the 32 nodes
// that follow its first.
constexpr int STATE_LEVEL = 18;  // where a family's state holds its leaves' level
constexpr uint32_t KID_LEAF = 0x80000000u;  // there are fewer than 2^29 elements
template <typename K>
__global__ void __launch_bounds__(256) k_node_children(const K *__restrict__ nodes, size_t nn, unsigned Lm,
                                                       uint2 *__restrict__ kids, uint8_t *__restrict__ leafs,
                                                       uint32_t *__restrict__ any) {
  typedef typename NodeWide<K>::W W;
  const int lane = threadIdx.x & 31;
  const size_t i0 = ((size_t)blockIdx.x * 256 + threadIdx.x) >> 5 << 2;
  if (i0 >= nn) return;
  const size_t i = i0 + (lane >> 3);
  const unsigned c = lane & 7;
  const W follow = i0 + 1 + lane < nn ? node_wide(nodes[i0 + 1 + lane]) : node_empty(W());
  const W k = i < nn ? node_wide(nodes[i]) : (W)0;
  const unsigned d = (unsigned)k & 31u;
  const W path = k >> 5;
  W ck = k + 1;  // level Lm: no node below
  if (d < Lm) ck = (path + ((W)c << (3 * (Lm - d - 1)))) << 5 | (W)(d + 1);
  int at = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (shfl_wide(follow, at + step - 1) < ck) at += step;
  const W found = shfl_wide(follow, at);
  size_t j = i0 + 1 + at;
  bool node = found == ck;
  if (i < nn && at == 31 && found < ck) {
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
  node = node && d < Lm;
  const unsigned leaf = __ballot_sync(0xffffffffu, i < nn && !node) >> (lane & 24) & 255u;
  if (i >= nn) return;
  kids[8 * i + c] = make_uint2((uint32_t)j | (node ? 0u : KID_LEAF),
                               (uint32_t)(7 * (j - (d + 1)) + digit_sum(path) + c));
  if (c == 0) {
    leafs[i] = (uint8_t)leaf;
    any[i] = leaf != 0;
  }
}

// the directions (as bits dx+1 + 3 (dy+1) + 9 (dz+1)) in which a leaf of the
// parent's size makes lattice point hang_pos(i) hang: away from the family
// along some of the axes on which the point lies on the parent's surface
__host__ __device__ constexpr uint32_t hang_dirs(int i) {
  const int d[3] = {hang_pos(i) % 3 - 1, hang_pos(i) / 3 % 3 - 1, hang_pos(i) / 9 - 1};
  uint32_t m = 0;
  for (int s = 1; s < 8; s++) {
    int t = 13;
    bool whole = true;
    for (int a = 0; a < 3; a++)
      if (s >> a & 1) {
        whole = whole && d[a] != 0;
        t += d[a] * (a == 0 ? 1 : a == 1 ? 3 : 9);
      }
    if (whole) m |= 1u << t;
  }
  return m;
}

// Elements, 8 threads per family (node f): thread q looks up the q-th parent
// of the family's 3x3x3 block; the family's neighbours are children of those,
// and those that are leaves hang lattice points.  Then thread c writes child
// c's element, if it is one, and its number of owned nodes.  block[8 f + q]
// keeps the parents for the lattices; state[f]: hanging points (18 bits),
// leaves' level (5), from bit 24 the children that are leaves.  list takes the families that have a
// leaf, in order (rank: how many before), which are those of the element loop.
template <typename K>
__global__ void __launch_bounds__(256) k_family_elems(const K *__restrict__ nodes, size_t nn, unsigned Lm,
                                                      const K *__restrict__ tab, const uint32_t *__restrict__ val,
                                                      uint64_t mask, const uint2 *__restrict__ kids,
                                                      const uint8_t *__restrict__ leafs,
                                                      const uint32_t *__restrict__ rank,
                                                      const uint8_t *__restrict__ etype_of,
                                                      uint32_t *__restrict__ block, uint32_t *__restrict__ state,
                                                      uint32_t *__restrict__ list,
                                                      uint32_t *__restrict__ meta, uint32_t *__restrict__ cnt,
                                                      uint32_t *flags) {
  typedef NodeWide<K> N;
  typedef typename N::W W;
  __shared__ int8_t bit_of[27];
  if (threadIdx.x < 27) bit_of[threadIdx.x] = (int8_t)hang_bit(threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, q8 = lane & 7, g0 = lane & 24;
  const size_t f = ((size_t)blockIdx.x * 256 + threadIdx.x) >> 3;
  const bool have = f < nn;
  const W k = have ? node_wide(nodes[f]) : (W)0;
  const unsigned d = (unsigned)k & 31u;
  uint32_t c[3];
  demorton3(N::key((k >> 5) >> (3 * (Lm - d))), c[0], c[1], c[2]);
  uint32_t ip = NODE_NONE;
  if (have && d > 0) {
    uint32_t par[3];
    bool in = true;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      par[a] = c[a] >> 1;
      if (q8 >> a & 1) {
        par[a] = (c[a] & 1u) ? par[a] + 1 : par[a] - 1;
        in = in && par[a] < 1u << (d - 1);  // -1 wraps round
      }
    }
    if (in) {
      const W key = N::of(morton3(par[0], par[1], par[2])) << (3 * (Lm - d + 1)) << 5 | (W)(d - 1);
      ip = node_find<K>(tab, val, mask, key, Lm);
    }
  }
  if (have) block[8 * f + q8] = ip;
  uint32_t leaf = 0;
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const int t = q8 + 8 * r;
    const int s[3] = {t % 3 - 1, t / 3 % 3 - 1, t / 9 - 1};
    int q = 0, digit = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (s[a] == ((c[a] & 1u) ? 1 : -1)) q |= 1 << a;
      digit |= (int)((c[a] + (uint32_t)s[a]) & 1u) << a;
    }
    const uint32_t iq = __shfl_sync(0xffffffffu, ip, g0 + q);
    if (t < 27 && t != 13 && iq != NODE_NONE && (leafs[iq] >> digit & 1u)) leaf |= 1u << t;
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) leaf |= __shfl_xor_sync(0xffffffffu, leaf, o);
  if (!have) return;
  uint32_t hang = 0;
#pragma unroll
  for (int i = 0; i < 18; i++)
    if (leaf & hang_dirs(i)) hang |= 1u << i;
  const uint32_t own = leafs[f];
  if (q8 == 0) {
    state[f] = hang | (d + 1) << STATE_LEVEL | own << 24;
    if (own) list[rank[f]] = (uint32_t)f;
  }
  if (!(own >> q8 & 1u)) return;
  const size_t e = kids[8 * f + q8].y;
  uint32_t hm = 0;
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const int b = bit_of[lat_vertex(q8, v)];
    if (b >= 0 && (hang >> b & 1u)) hm |= 1u << v;
  }
  uint32_t et = etype_of[q8 * 256 + hm];
  if (et == 0xffu) {
    set_flag(flags, DGF_NOT_BALANCED);
    et = 0;
  }
  meta[e] = (d + 1) | (uint32_t)q8 << 8 | hm << 16 | et << 24;
  unsigned bdy = 0, owned = 0;
#pragma unroll
  for (int a = 0; a < 3; a++)
    if (2 * c[a] + (q8 >> a & 1) + 1 == 2u << d) bdy |= 1u << a;
#pragma unroll
  for (int v = 0; v < 8; v++)
    if ((v & bdy) == (unsigned)v && !(hm >> v & 1u)) owned++;
  cnt[e] = owned;
}

// ------------------------------------------------------------------------
// connectivity and element loop tables: the lattices of the families, and the
// nodes of each patch of families (layout: dg_elem.cuh)
// ------------------------------------------------------------------------
// Lattices, 8 threads per family: the mesh node at a lattice point is owned by
// the element anchored there, a child of the family or of its neighbour in
// positive directions (on the domain's positive boundary the leaf inside, by a
// search).  The parents, children and their elements come from the 8 lanes by
// shuffles; a lane's points go through three dependent loads side by side, and
// the rare searches follow.  From the lattices the elements' node ids, if
// wanted, and the coordinates of the nodes that they own.  A kernel of its own,
// for the loads in flight: inside the patch kernel, with the registers and
// shared memory of that, the two took 0.72 ms together (1e6-point mesh).
// lat: [patch][point][family], NO_NODE where no element refers to the point.
constexpr uint32_t NO_NODE = 0xffffffffu;
constexpr int LF_BLOCK = 256, LF_FAM = LF_BLOCK / 8;
static_assert(FAM % LF_FAM == 0, "a block's families lie in one patch");

template <typename K>
__global__ void __launch_bounds__(LF_BLOCK)
    k_family_lattice(const K *__restrict__ nodes, const uint32_t *__restrict__ list, size_t n_fam, unsigned Lm,
                     unsigned D, const Key128 *__restrict__ keys, size_t n, const uint2 *__restrict__ kids,
                     const uint32_t *__restrict__ block, const uint32_t *__restrict__ state,
                     const uint32_t *__restrict__ meta, const uint32_t *__restrict__ base, size_t n_node,
                     uint32_t *__restrict__ conn, uint32_t *__restrict__ nx, uint32_t *__restrict__ ny,
                     uint32_t *__restrict__ nz, uint32_t *__restrict__ lat, uint32_t *flags) {
  typedef NodeWide<K> N;
  __shared__ uint32_t s_lat[27][LF_FAM + 1];
  __shared__ int8_t bit_of[27];
  const int t = threadIdx.x, q8 = t & 7, g0 = t & 24, at = t >> 3;
  if (t < 27) bit_of[t] = (int8_t)hang_bit(t);
  __syncthreads();
  const size_t r = (size_t)blockIdx.x * LF_FAM + at;
  const bool have = r < n_fam;
  const size_t f = have ? list[r] : 0;
  const auto k = node_wide(nodes[f]);
  const unsigned d = (unsigned)k & 31u;
  uint32_t c[3];
  demorton3(N::key((k >> 5) >> (3 * (Lm - d))), c[0], c[1], c[2]);
  const uint32_t st = have ? state[f] : 0u, hang = st & 0x3ffffu;
  const bool leaf = st >> 24 >> q8 & 1u;
  const unsigned sh = D - d - 1;  // lattice spacing 2^sh
  const uint32_t e = kids[8 * f + q8].y, par = block[8 * f + q8];
  // the points that the family's elements refer to
  uint32_t used = 0, hm = 0;
  if (leaf) {
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const int pos = lat_vertex(q8, v), b = bit_of[pos];
      const bool h = b >= 0 && (hang >> b & 1u);
      used |= 1u << (h ? lat_corner(v) : pos);
      hm |= (uint32_t)h << v;
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) used |= __shfl_xor_sync(0xffffffffu, used, o);
  // the owners of points q8, q8 + 8, ...
  uint32_t own[4];
  unsigned search = 0, ok = 15u;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int i = q8 + 8 * j;
    const int pt[3] = {i % 3, i / 3 % 3, i / 9};
    int q = 0, digit = 0, child = 0;
    bool out = false, edge = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (pt[a] == 2) {
        out = true;
        edge = edge || c[a] + 1 == 1u << d;
        if (c[a] & 1u) q |= 1 << a;
      }
      digit |= (int)((c[a] + (pt[a] == 2 ? 1u : 0u)) & 1u) << a;
      child |= (pt[a] & 1) << a;
    }
    const uint32_t iq = __shfl_sync(0xffffffffu, par, g0 + q);
    own[j] = __shfl_sync(0xffffffffu, e, g0 + child);
    if (i < 27 && (used >> i & 1u) && out) {
      if (edge || iq == NODE_NONE) {  // no such parent: a leaf two levels up, perhaps anchored here
        search |= 1u << j;
      } else {
        const uint2 kid = kids[8 * (size_t)iq + digit];
        own[j] = kid.y;  // the leaf, or the first below the node
        if (child) {
          if (kid.x & KID_LEAF) ok &= ~(1u << j);
          else own[j] = kids[8 * (size_t)kid.x + child].y;
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int i = q8 + 8 * j;
    uint32_t id = NO_NODE;
    if (i < 27 && (used >> i & 1u) && !(search >> j & 1u)) {
      id = base[own[j]];
      if (!(ok >> j & 1u) || (meta[own[j]] >> 16 & 1u) || id >= n_node) {
        set_flag(flags, DGF_NOT_BALANCED);
        id = 0;
      }
    }
    if (i < 27) s_lat[i][at] = id;
  }
  const uint32_t e0 = __shfl_sync(0xffffffffu, e, g0);
  while (search) {
    // the leaf that contains the point, moved inside the domain
    const int i = q8 + 8 * (__ffs(search) - 1);
    search &= search - 1;
    const int pt[3] = {i % 3, i / 3 % 3, i / 9};
    int kb = 0, bo = 0;
    uint32_t v[3], cl[3], oc[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      v[a] = (2 * c[a] + (uint32_t)pt[a]) << sh;
      if (pt[a] == 2 && c[a] + 1 == 1u << d) kb |= 1 << a;
      cl[a] = (kb >> a & 1) ? v[a] - 1 : v[a];
    }
    const size_t o = find_leaf_from(keys, n, morton3(cl[0], cl[1], cl[2]), e0);
    const Key128 ko = keys[o];
    const uint32_t ho = 1u << (D - tag_level(ko));
    demorton3(tag_anchor(ko), oc[0], oc[1], oc[2]);
    bool good = true;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      good = good && ((kb >> a & 1) ? oc[a] + ho == 1u << D : oc[a] == v[a]);
      if (oc[a] + ho == 1u << D) bo |= 1 << a;
    }
    const unsigned hmo = meta[o] >> 16 & 255u;
    unsigned before = 0;  // nodes that it owns before this one
    for (int s = 0; s < kb; s++)
      if ((s & bo) == s && !(hmo >> s & 1u)) before++;
    uint32_t id = base[o] + before;
    if (!good || (hmo >> kb & 1u) || id >= n_node) {
      set_flag(flags, DGF_NOT_BALANCED);
      id = 0;
    }
    s_lat[i][at] = id;
  }
  __syncthreads();
  // a warp writes a point of the block's 32 families
  const size_t r0 = (size_t)blockIdx.x * LF_FAM;
  uint32_t *row = lat + r0 / FAM * (27 * FAM) + r0 % FAM + (t & 31);
  for (int i = t >> 5; i < 27; i += LF_BLOCK / 32) row[(size_t)i * FAM] = s_lat[i][t & 31];
  if (!leaf) return;
  if (conn)
#pragma unroll
    for (int v = 0; v < 8; v++)
      conn[(size_t)v * n + e] = s_lat[(hm >> v & 1u) ? lat_corner(v) : lat_vertex(q8, v)][at];
  unsigned bdy = 0;
  uint32_t x[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const uint32_t g = 2 * c[a] + (q8 >> a & 1);
    x[a] = g << sh;
    if (g + 1 == 2u << d) bdy |= 1u << a;
  }
  uint32_t id = base[e];
  for (unsigned v = 0; v < 8; v++) {
    if ((v & bdy) != v || (hm >> v & 1u)) continue;
    if (id < n_node) {
      nx[id] = x[0] + ((v & 1u) << sh);
      ny[id] = x[1] + ((v >> 1 & 1u) << sh);
      nz[id] = x[2] + ((v >> 2) << sh);
    }
    id++;
  }
}

// ------------------------------------------------------------------------
// any other records: element by element
// ------------------------------------------------------------------------
// Records that are not the leaves of a complete octree in order (a leaf that
// no vertex refers to may be missing, elements may stand in another order) and
// the octree that is one element have no nodes to start from.  Elements are
// found by their anchors in a hash table over all of them instead.  Such
// records are a mesh if every vertex finds its owner.
// linear probing over a power-of-two table of element indices (at most half
// full); a slot's anchor is read back from the keys.
constexpr uint32_t AH_EMPTY = 0xffffffffu;

__device__ __forceinline__ uint64_t anchor_hash(Key128 a) {
  uint64_t x = a.lo ^ (a.hi * 0x9e3779b97f4a7c15ull);
  x ^= x >> 31;
  x *= 0xbf58476d1ce4e5b9ull;
  x ^= x >> 29;
  return x;
}

__global__ void k_anchor_insert(const Key128 *__restrict__ keys, size_t n, uint32_t *__restrict__ tab, uint64_t mask) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  uint64_t h = anchor_hash(tag_anchor(keys[e])) & mask;
  for (uint64_t probe = 0; probe <= mask; probe++) {
    if (atomicCAS(&tab[h], AH_EMPTY, (uint32_t)e) == AH_EMPTY) return;
    h = (h + 1) & mask;
  }
}

// element anchored at `pos` (a bare anchor), or AH_EMPTY
__device__ __forceinline__ uint32_t anchor_find(const Key128 *__restrict__ keys, const uint32_t *__restrict__ tab,
                                                uint64_t mask, Key128 pos) {
  uint64_t h = anchor_hash(pos) & mask;
  for (uint64_t probe = 0; probe <= mask; probe++) {
    const uint32_t e = tab[h];
    if (e == AH_EMPTY) return AH_EMPTY;
    if (key_eq(tag_anchor(keys[e]), pos)) return e;
    h = (h + 1) & mask;
  }
  return AH_EMPTY;
}

__device__ __forceinline__ bool is_leaf_at(const Key128 *__restrict__ keys, const uint32_t *__restrict__ tab,
                                           uint64_t mask, int64_t x, int64_t y, int64_t z, unsigned lev, int64_t dom) {
  if (x < 0 || y < 0 || z < 0 || x >= dom || y >= dom || z >= dom) return false;
  const uint32_t j = anchor_find(keys, tab, mask, morton3((uint32_t)x, (uint32_t)y, (uint32_t)z));
  return j != AH_EMPTY && tag_level(keys[j]) == lev;
}

__global__ void k_mesh_elems(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                             uint64_t mask, unsigned D, const uint8_t *__restrict__ etype_of,
                             uint32_t *__restrict__ meta, uint32_t *__restrict__ cnt, uint32_t *flags) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const unsigned l = tag_level(ke);
  uint32_t ux, uy, uz;
  demorton3(tag_anchor(ke), ux, uy, uz);
  const int64_t dom = (int64_t)1 << D, h = (int64_t)1 << (D - l);
  const int64_t x = ux, y = uy, z = uz;
  int c = 0;
  if (l > 0) c = (int)(((x >> (D - l)) & 1) | (((y >> (D - l)) & 1) << 1) | (((z >> (D - l)) & 1) << 2));
  unsigned hm = 0;
  if (l > 1) {
    const int64_t H = 2 * h;
    const int64_t P[3] = {x - ((c & 1) ? h : 0), y - ((c & 2) ? h : 0), z - ((c & 4) ? h : 0)};
    const int64_t d[3] = {(c & 1) ? H : -H, (c & 2) ? H : -H, (c & 4) ? H : -H};
    // neighbours of P towards the child's exterior: leaf[s] for s in 1..7
    bool leaf[8];
    leaf[0] = false;
#pragma unroll
    for (int s = 1; s < 8; s++) {
      if (s == 7) {
        leaf[s] = false;  // the corner neighbour hangs no vertex of e
        continue;
      }
      leaf[s] = is_leaf_at(keys, tab, mask, P[0] + ((s & 1) ? d[0] : 0), P[1] + ((s & 2) ? d[1] : 0),
                           P[2] + ((s & 4) ? d[2] : 0), l - 1, dom);
    }
#pragma unroll
    for (int r = 1; r < 7; r++) {
      const int others = 7 & ~r;
      bool hang = false;
#pragma unroll
      for (int s = 1; s < 7; s++)
        if ((s & others) == s && leaf[s]) hang = true;
      if (hang) hm |= 1u << (c ^ r);
    }
  }
  unsigned et = etype_of[c * 256 + hm];
  if (et == 0xffu) {
    set_flag(flags, DGF_NOT_BALANCED);
    et = 0;
  }
  meta[e] = l | ((unsigned)c << 8) | (hm << 16) | (et << 24);
  const unsigned bdy = ((x + h == dom) ? 1u : 0u) | ((y + h == dom) ? 2u : 0u) | ((z + h == dom) ? 4u : 0u);
  unsigned owned = 0;
#pragma unroll
  for (int k = 0; k < 8; k++)
    if ((k & bdy) == (unsigned)k && !(hm >> k & 1)) owned++;
  cnt[e] = owned;
}

__global__ void k_mesh_conn(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                            uint64_t mask, unsigned D, const uint32_t *__restrict__ meta,
                            const uint32_t *__restrict__ base, uint32_t *__restrict__ conn, uint32_t *__restrict__ nx,
                            uint32_t *__restrict__ ny, uint32_t *__restrict__ nz, size_t n_node, uint32_t *flags) {
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const uint32_t me = meta[e];
  const unsigned l = me & 255u, c = (me >> 8) & 7u, hm = (me >> 16) & 255u;
  uint32_t ux, uy, uz;
  demorton3(tag_anchor(ke), ux, uy, uz);
  const int64_t dom = (int64_t)1 << D, h = (int64_t)1 << (D - l);
  const int64_t x = ux, y = uy, z = uz;
  const int64_t px = x - ((c & 1) ? h : 0), py = y - ((c & 2) ? h : 0), pz = z - ((c & 4) ? h : 0);
  // owned nodes: coordinates
  {
    const unsigned bdy = ((x + h == dom) ? 1u : 0u) | ((y + h == dom) ? 2u : 0u) | ((z + h == dom) ? 4u : 0u);
    uint64_t id = base[e];
    for (int k = 0; k < 8; k++) {
      if ((k & bdy) != (unsigned)k || (hm >> k & 1)) continue;
      if (id < n_node) {
        nx[id] = (uint32_t)(x + ((k & 1) ? h : 0));
        ny[id] = (uint32_t)(y + ((k & 2) ? h : 0));
        nz[id] = (uint32_t)(z + ((k & 4) ? h : 0));
      }
      id++;
    }
  }
#pragma unroll 1
  for (int k = 0; k < 8; k++) {
    int64_t v[3];
    if (hm >> k & 1) {
      v[0] = px + ((k & 1) ? 2 * h : 0);
      v[1] = py + ((k & 2) ? 2 * h : 0);
      v[2] = pz + ((k & 4) ? 2 * h : 0);
    } else {
      v[0] = x + ((k & 1) ? h : 0);
      v[1] = y + ((k & 2) ? h : 0);
      v[2] = z + ((k & 4) ? h : 0);
    }
    unsigned kb = 0;
    int64_t cl[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (v[a] == dom) {
        kb |= 1u << a;
        cl[a] = dom - 1;
      } else {
        cl[a] = v[a];
      }
    }
    // the owner is the element anchored at the vertex; on the positive domain
    // boundary, the leaf containing the vertex clamped inward (a search)
    size_t o;
    bool found = true;
    if (k == 0 && !(hm & 1u)) {
      o = e;  // a vertex 0 that does not hang is the element's own anchor
    } else if (kb == 0) {
      const uint32_t f = anchor_find(keys, tab, mask, morton3((uint32_t)cl[0], (uint32_t)cl[1], (uint32_t)cl[2]));
      found = f != AH_EMPTY;
      o = found ? f : 0;
    } else {
      o = find_leaf_from(keys, n, morton3((uint32_t)cl[0], (uint32_t)cl[1], (uint32_t)cl[2]), e);
    }
    const Key128 ko = keys[o];
    const unsigned lo_ = tag_level(ko);
    const int64_t ho = (int64_t)1 << (D - lo_);
    // the owner's anchor: the vertex itself when it was found by its anchor
    // (no decode needed), else decoded from the owner's key
    int64_t oc[3] = {v[0], v[1], v[2]};
    bool ok = found;
    if (kb != 0) {
      uint32_t ox, oy, oz;
      demorton3(tag_anchor(ko), ox, oy, oz);
      oc[0] = ox;
      oc[1] = oy;
      oc[2] = oz;
#pragma unroll
      for (int a = 0; a < 3; a++) ok = ok && ((kb >> a & 1) ? (oc[a] + ho == dom) : (oc[a] == v[a]));
    }
    const unsigned bo = ((oc[0] + ho == dom) ? 1u : 0u) | ((oc[1] + ho == dom) ? 2u : 0u) | ((oc[2] + ho == dom) ? 4u : 0u);
    const unsigned hmo = (meta[o] >> 16) & 255u;
    ok = ok && ((kb & bo) == kb) && !(hmo >> kb & 1);
    unsigned rank = 0;
    for (unsigned q = 0; q < kb; q++)
      if ((q & bo) == q && !(hmo >> q & 1)) rank++;
    uint64_t id = base[o] + rank;
    if (!ok || id >= n_node) {
      set_flag(flags, DGF_NOT_BALANCED);
      id = 0;
    }
    conn[(size_t)k * n + e] = (uint32_t)id;
  }
}

// a family's first element: the lowest child of its parent that is a leaf
// (children before e: e - 1 in the usual case, else look-ups)
__global__ void k_family_heads(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab,
                               uint64_t mask, unsigned D, uint32_t *__restrict__ head) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const Key128 ke = keys[e];
  const unsigned l = tag_level(ke);
  bool first = true;
  if (l > 0) {
    const Key128 a = tag_anchor(ke);
    const unsigned sh = 3 * (D - l);
    const unsigned c = (unsigned)(key_shr(a, sh).lo & 7u);
    if (c > 0 && e > 0) {
      const Key128 kp = keys[e - 1];
      first = !(tag_level(kp) == l && key_eq(key_shr(tag_anchor(kp), sh + 3), key_shr(a, sh + 3)));
      if (first) {
        for (unsigned q = 0; q < c && first; q++) {
          const uint32_t j =
              anchor_find(keys, tab, mask, key_xor(a, key_shl(Key128{(uint64_t)(q ^ c), 0}, sh)));
          first = !(j != AH_EMPTY && tag_level(keys[j]) == l);
        }
      }
    }
  }
  head[e] = first ? 1u : 0u;
}

__global__ void k_family_list(const uint32_t *__restrict__ head, const uint32_t *__restrict__ pos, size_t n,
                              uint32_t *__restrict__ first) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n && head[e]) first[pos[e]] = (uint32_t)e;
}

// family f's children (the element after a child is its next sibling, or a
// look-up tells), its state and its lattice from the elements' node ids
__global__ void __launch_bounds__(FAM)
    k_leaf_lattice(const Key128 *__restrict__ keys, size_t n, const uint32_t *__restrict__ tab, uint64_t tmask,
                   unsigned D, const uint32_t *__restrict__ first, size_t n_fam, const uint32_t *__restrict__ meta,
                   const uint32_t *__restrict__ conn, uint32_t *__restrict__ list, uint2 *__restrict__ kids,
                   uint32_t *__restrict__ state, uint32_t *__restrict__ lattice) {
  const size_t p = blockIdx.x, f = p * FAM + threadIdx.x;
  uint32_t el[8], mask = 0;
#pragma unroll
  for (int c = 0; c < 8; c++) el[c] = 0;
  if (f < n_fam) {
    const uint32_t e0 = first[f];
    const Key128 a = tag_anchor(keys[e0]);
    const unsigned l = tag_level(keys[e0]);
    if (l == 0) {
      el[0] = e0;
      mask = 1;
    } else {
      const unsigned sh = 3 * (D - l);
      const unsigned c0 = (unsigned)(key_shr(a, sh).lo & 7u);
      const Key128 par = key_shr(a, sh + 3);
      uint32_t prev = e0;
#pragma unroll
      for (unsigned c = 0; c < 8; c++) {
        if (c < c0) continue;
        uint32_t e = c == c0 ? e0 : prev + 1;
        bool ok = c == c0;
        if (!ok && e < n) {
          const Key128 k = keys[e];
          const Key128 s = key_shr(tag_anchor(k), sh);
          ok = tag_level(k) == l && (unsigned)(s.lo & 7u) == c && key_eq(key_shr(s, 3), par);
        }
        if (!ok) {
          e = anchor_find(keys, tab, tmask, key_xor(a, key_shl(Key128{(uint64_t)(c ^ c0), 0}, sh)));
          ok = e != AH_EMPTY && tag_level(keys[e]) == l;
        }
        if (ok) {
          el[c] = e;
          mask |= 1u << c;
          prev = e;
        }
      }
    }
  }
  uint32_t lat[27], hang = 0, lev = 0;
#pragma unroll
  for (int i = 0; i < 27; i++) lat[i] = NO_NODE;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (!(mask >> c & 1u)) continue;
    const uint32_t me = meta[el[c]];
    lev = me & 255u;
    const uint32_t hm = me >> 16 & 255u;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int bit = hang_bit(lat_vertex(c, k));
      if (bit >= 0 && (hm >> k & 1u)) {
        hang |= 1u << (bit & 31);
        if (lat[lat_corner(k)] == NO_NODE) lat[lat_corner(k)] = conn[(size_t)k * n + el[c]];
      } else if (lat[lat_vertex(c, k)] == NO_NODE) {
        lat[lat_vertex(c, k)] = conn[(size_t)k * n + el[c]];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 27; i++) lattice[(p * 27 + i) * FAM + threadIdx.x] = lat[i];
  if (f >= n_fam) return;
  list[f] = (uint32_t)f;
  state[f] = hang | lev << STATE_LEVEL | mask << 24;
#pragma unroll
  for (int c = 0; c < 8; c++) kids[8 * f + c] = make_uint2(0u, el[c]);
}

// ------------------------------------------------------------------------
// patch tables
// ------------------------------------------------------------------------
// The patches' tables, one block per patch: complete families move to the
// front, and the nodes are numbered through a shared-memory hash table.  The
// nodes are numbered in claim order, for the element loop's shared-memory banks
// (number mod 32; shared FP32 atomic adds at random banks cost about four times
// those at distinct banks, measured 13.7 against 3.3 cycles per warp
// instruction on an SM): the nodes that a warp claims at one lattice point take
// consecutive numbers, so they fall on distinct banks when that warp touches
// them together.  Patches append their nodes to one list (any order).
constexpr int PF_HT = 4096;  // hash slots, more than FAM_MAX_RUN
static_assert(FAM_MAX_RUN < PF_HT, "a patch's nodes must fit the hash table");

struct PatchFamSmem {
  uint32_t hkey[PF_HT];          // node of each hash slot
  uint32_t node[FAM_MAX_RUN];    // node of each number
  uint16_t num[PF_HT];           // number of each hash slot
  uint8_t order[FAM];            // family at each place
  int counter;
  unsigned long long base;
};

__global__ void __launch_bounds__(FAM)
    k_patch_families(const uint32_t *__restrict__ list, size_t n_fam, const uint2 *__restrict__ kids,
                     const uint32_t *__restrict__ state, const uint32_t *__restrict__ lattice, uint4 *__restrict__ fam, uint4 *__restrict__ pinfo,
                     uint32_t *__restrict__ fchild, uint32_t *__restrict__ run_node,
                     uint32_t *__restrict__ node_patches, unsigned long long *__restrict__ n_run,
                     uint32_t *__restrict__ max_run) {
  extern __shared__ __align__(16) unsigned char pf_raw[];
  PatchFamSmem &S = *reinterpret_cast<PatchFamSmem *>(pf_raw);
  const int t = threadIdx.x, lane = t & 31;
  const size_t p = blockIdx.x;
  for (int i = t; i < PF_HT; i += FAM) S.hkey[i] = NO_NODE;
  if (t == 0) S.counter = 0;
  __syncthreads();
  // 1. complete families first
  {
    const size_t r = p * FAM + t;
    const bool whole = r < n_fam && state[list[r]] >> 24 == 255u;
    int n_whole;
    const int before = block_excl_scan<int, FAM>(whole ? 1 : 0, n_whole);
    S.order[whole ? before : n_whole + (t - before)] = (uint8_t)t;
  }
  __syncthreads();
  // 2. this place's family
  const int from = S.order[t];
  uint32_t lat[27], mask = 0, hang = 0, lev = 0;
#pragma unroll
  for (int i = 0; i < 27; i++) lat[i] = lattice[(p * 27 + i) * FAM + from];
  if (p * FAM + from < n_fam) {
    const size_t f = list[p * FAM + from];
    mask = state[f] >> 24;
    hang = state[f] & 0x3ffffu;
    lev = state[f] >> STATE_LEVEL & 31u;
    uint4 *fc = reinterpret_cast<uint4 *>(fchild + 8 * (p * FAM + t));
    uint4 el[4];
#pragma unroll
    for (int q = 0; q < 4; q++) el[q] = reinterpret_cast<const uint4 *>(kids + 8 * f)[q];
    fc[0] = make_uint4(el[0].y, el[0].w, el[1].y, el[1].w);
    fc[1] = make_uint4(el[2].y, el[2].w, el[3].y, el[3].w);
  }
  // 3. number the nodes
  uint16_t slot[27];
#pragma unroll
  for (int i = 0; i < 27; i++) {
    const uint32_t g = lat[i];
    uint32_t h = (g * 2654435761u) >> (32 - 12);  // PF_HT = 2^12
    bool won = false;
    if (g != NO_NODE) {
      for (int probe = 0; probe < PF_HT; probe++) {
        const uint32_t cur = atomicCAS(&S.hkey[h], NO_NODE, g);
        won = cur == NO_NODE;
        if (won || cur == g) break;
        h = (h + 1) & (PF_HT - 1);
      }
    }
    slot[i] = (uint16_t)h;
    const unsigned claims = __ballot_sync(0xffffffffu, won);
    if (claims) {
      const int leader = __ffs(claims) - 1;
      int at0 = 0;
      if (lane == leader) at0 = atomicAdd(&S.counter, __popc(claims));
      at0 = __shfl_sync(0xffffffffu, at0, leader);
      if (won) {
        const int u = at0 + __popc(claims & ((1u << lane) - 1u));
        S.num[h] = (uint16_t)(u + 1);
        S.node[u] = g;
      }
    }
  }
  __syncthreads();
  const int nr = S.counter;
  if (t == 0) {
    S.base = atomicAdd(n_run, (unsigned long long)nr);
    atomicMax(max_run, (uint32_t)nr);
    pinfo[p] = make_uint4((uint32_t)S.base, (uint32_t)(S.base >> 32), (uint32_t)nr, 0u);
  }
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; i++) w[i] = 0;
#pragma unroll
  for (int i = 0; i < 27; i++)
    if (lat[i] != NO_NODE) w[i >> 1] |= (uint32_t)S.num[slot[i]] << (i & 1 ? 16 : 0);
  w[13] |= lev << 16;
  w[14] = mask | (hang & 0xffffu) << 16;
  w[15] = hang >> 16;
#pragma unroll
  for (int q = 0; q < 4; q++)
    fam[(p * 4 + q) * FAM + t] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  __syncthreads();
  for (int u = t; u < nr; u += FAM) {
    const uint32_t g = S.node[u];
    run_node[S.base + u] = g;
    atomicAdd(&node_patches[g], 1u);
  }
}

// the run words: node, "no other patch touches it", "on the domain boundary"
__global__ void k_run_flags(const uint32_t *__restrict__ run_node, size_t n_run,
                            const uint32_t *__restrict__ node_patches, const uint32_t *__restrict__ node_xyz, size_t V,
                            uint32_t dom, uint32_t *__restrict__ prun) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_run) return;
  const uint32_t g = run_node[i];
  const uint32_t x = node_xyz[g], y = node_xyz[V + g], z = node_xyz[2 * V + g];
  const bool bdy = x == 0 || y == 0 || z == 0 || x == dom || y == dom || z == dom;
  prun[i] = g | (node_patches[g] == 1u ? PRUN_COMPLETE : 0u) | (bdy ? PRUN_BDY : 0u);
}

// conn from the family tables: child c's vertex k is its lattice point, or
// the parent's corner k where that point hangs
__global__ void __launch_bounds__(FAM) k_conn_from_families(const uint4 *__restrict__ fam,
                                                            const uint4 *__restrict__ pinfo,
                                                            const uint32_t *__restrict__ prun,
                                                            const uint32_t *__restrict__ fchild, size_t n_fam,
                                                            size_t E, uint32_t *__restrict__ conn) {
  const size_t p = blockIdx.x;
  const int t = threadIdx.x;
  if (p * FAM + t >= n_fam) return;
  const uint4 info = pinfo[p];
  const uint32_t *run = prun + ((size_t)info.x | (size_t)info.y << 32);
  uint4 w[4];
#pragma unroll
  for (int q = 0; q < 4; q++) w[q] = fam[(p * 4 + q) * FAM + t];
  const uint32_t mask = fam_mask(w), hang = fam_hang(w);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    if (!(mask >> c & 1u)) continue;
    const size_t e = fchild[8 * (p * FAM + t) + c];
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int bit = hang_bit(lat_vertex(c, k));
      const bool h = bit >= 0 && (hang >> (bit & 31) & 1u);
      const uint32_t u = h ? fam_u16(w, lat_corner(k)) : fam_u16(w, lat_vertex(c, k));
      conn[(size_t)k * E + e] = run[u - 1] & PRUN_NODE;
    }
  }
}

const uint32_t *mesh_conn(Context &ctx, const Mesh &m, DBuf<uint32_t> &tmp) {
  if (!m.compressed) return m.conn;
  tmp.alloc(8 * m.n_elem, ctx.stream);
  ProfScope _prof(ctx, "da_conn_decode", (double)m.n_elem * 32 + (double)m.n_fam * 96 + (double)m.n_run * 4);
  k_conn_from_families<<<(unsigned)m.n_patch, FAM, 0, ctx.stream>>>(m.fam, m.pinfo, m.prun, m.fchild, m.n_fam,
                                                                    m.n_elem, tmp.get());
  DG_LAUNCH_CHECK();
  return tmp.get();
}

size_t mesh_bytes(const Mesh &m) {
  size_t b = m.n_elem * 4 + m.n_node * 12;  // meta, node coordinates
  if (m.conn) b += 8 * m.n_elem * 4;
  b += m.n_patch * (4 * FAM + 1) * sizeof(uint4) + m.n_run * 4 + m.n_fam * 32;  // family tables
  return b;
}

// the element loop's tables of a mesh whose nodes are numbered; its families'
// elements, states and lattices are given
static void mesh_patches(Context &ctx, Mesh &m, const uint32_t *list, size_t nf, const uint2 *kids,
                         const uint32_t *state, const uint32_t *lat) {
  cudaStream_t s = ctx.stream;
  const size_t nn = m.n_node, np = (nf + FAM - 1) / FAM;
  DBuf<uint32_t> fchild(8 * nf, s), run_node(27 * nf, s), npatch(nn ? nn : 1, s);
  DBuf<uint4> fam(np * 4 * FAM, s), pinfo(np, s);
  DG_CUDA(cudaMemsetAsync(npatch.get(), 0, nn * sizeof(uint32_t), s));
  unsigned long long *d_run = ctx.d_scratch;  // {nodes of all patches, most of one}
  DG_CUDA(cudaMemsetAsync(d_run, 0, 2 * sizeof(unsigned long long), s));
  {
    ProfScope _prof(ctx, "da_patch_families", (double)nf * (108 + 64 + 100) + (double)nn * 8);
    ensure_smem_attr(ctx, k_patch_families, (int)sizeof(PatchFamSmem));
    k_patch_families<<<(unsigned)np, FAM, sizeof(PatchFamSmem), s>>>(
        list, nf, kids, state, lat, fam.get(), pinfo.get(), fchild.get(), run_node.get(), npatch.get(), d_run,
        reinterpret_cast<uint32_t *>(d_run + 1));
    DG_LAUNCH_CHECK();
  }
  DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_run, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
  check_device_flags(ctx, "DA");
  const size_t nruns = (size_t)ctx.h_scratch[4];
  m.max_run = (int)(uint32_t)ctx.h_scratch[5];
  DBuf<uint32_t> prun(nruns ? nruns : 1, s);
  {
    ProfScope _prof(ctx, "da_run_flags", (double)nruns * 24);
    k_run_flags<<<grid_for(nruns, 256), 256, 0, s>>>(run_node.get(), nruns, npatch.get(), m.node_xyz, nn,
                                                     1u << m.max_depth, prun.get());
    DG_LAUNCH_CHECK();
  }
  m.n_fam = nf;
  m.n_patch = np;
  m.n_run = nruns;
  m.fam = fam.release_ptr();
  m.pinfo = pinfo.release_ptr();
  m.prun = prun.release_ptr();
  m.fchild = fchild.release_ptr();
}

template <typename K>
static void build_from_nodes(Context &ctx, const Octree &bal, const Octree &tree, Mesh &m) {
  cudaStream_t s = ctx.stream;
  const size_t n = bal.n, n_int = tree.n_node;
  const unsigned D = bal.max_depth, Lm = tree.top - 1;
  const K *nodes = static_cast<const K *>(tree.nodes);
  DBuf<K> tab;
  DBuf<uint32_t> val, rank(n_int, s), block(8 * n_int, s), state(n_int, s), list(n_int, s);
  DBuf<uint2> kids(8 * n_int, s);
  DBuf<uint8_t> leafs(n_int, s);
  DBuf<uint32_t> meta(n, s), base(n, s);
  uint32_t *d_total = reinterpret_cast<uint32_t *>(ctx.d_scratch);  // {families with a leaf, mesh nodes}
  {
    ProfScope _prof(ctx, "da_node_children", (double)n_int * (sizeof(K) + 69));
    k_node_children<K><<<grid_for(8 * n_int, 256), 256, 0, s>>>(nodes, n_int, Lm, kids.get(), leafs.get(),
                                                                rank.get());
    DG_LAUNCH_CHECK();
  }
  exclusive_scan<uint32_t, uint32_t>(rank.get(), rank.get(), n_int, d_total, s);
  size_t slots = 1024;
  while (slots < 2 * n_int) slots <<= 1;
  for (;; slots *= 2) {  // again where a node found no slot
    tab.alloc(slots, s);
    val.alloc(slots, s);
    DG_CUDA(cudaMemsetAsync(tab.get(), 0xff, slots * sizeof(K), s));
    DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
    {
      ProfScope _prof(ctx, "da_node_table", (double)n_int * (2 * sizeof(K) + 4));
      k_node_table<K><<<grid_for(n_int, 256), 256, 0, s>>>(nodes, n_int, Lm, tab.get(), val.get(), slots - 1,
                                                           ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    {
      ProfScope _prof(ctx, "da_elems", (double)n_int * (sizeof(K) + 77) + (double)n * 8);
      k_family_elems<K><<<grid_for(8 * n_int, 256), 256, 0, s>>>(
          nodes, n_int, Lm, tab.get(), val.get(), slots - 1, kids.get(), leafs.get(), rank.get(), ctx.d_etype_of,
          block.get(), state.get(), list.get(), meta.get(), base.get(), ctx.d_flags);
      DG_LAUNCH_CHECK();
    }
    exclusive_scan<uint32_t, uint32_t>(base.get(), base.get(), n, d_total + 1, s);
    DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_total, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    const uint32_t f = read_scalar(ctx, ctx.d_flags);
    if (f & DGF_CAPACITY) continue;
    if (f) check_device_flags(ctx, "DA");
    break;
  }
  uint32_t total[2];
  std::memcpy(total, ctx.h_scratch + 4, sizeof(total));
  const size_t nf = total[0], nn = total[1], np = (nf + FAM - 1) / FAM;
  if (nn >= (size_t)PRUN_BDY) fail(DG_ERR_INVALID_ARG, "DA: too many nodes for the element loop tables");
  DBuf<uint32_t> conn, nxyz(3 * (nn ? nn : 1), s), lat(np * 27 * FAM, s);
  if (!m.compressed) conn.alloc(8 * n, s);
  {
    ProfScope _prof(ctx, "da_lattices", (double)n * (8 + (m.compressed ? 0 : 32)) + (double)nn * 12 + (double)nf * 220);
    k_family_lattice<K><<<(unsigned)(np * (FAM / LF_FAM)), LF_BLOCK, 0, s>>>(
        nodes, list.get(), nf, Lm, D, bal.keys, n, kids.get(), block.get(), state.get(), meta.get(), base.get(), nn,
        conn.get(), nxyz.get(), nxyz.get() + nn, nxyz.get() + 2 * nn, lat.get(), ctx.d_flags);
    DG_LAUNCH_CHECK();
  }
  m.n_node = nn;
  m.node_xyz = nxyz.release_ptr();
  m.conn = conn.release_ptr();
  m.meta = meta.release_ptr();
  mesh_patches(ctx, m, list.get(), nf, kids.get(), state.get(), lat.get());
}

static void build_from_leaves(Context &ctx, const Octree &bal, Mesh &m) {
  cudaStream_t s = ctx.stream;
  const size_t n = bal.n;
  const unsigned D = bal.max_depth;
  DBuf<uint32_t> meta(n, s), base(n, s), head(n, s), pos(n, s);
  size_t cap = 1;
  while (cap < 2 * n) cap <<= 1;
  DBuf<uint32_t> atab(cap, s);
  const uint64_t amask = cap - 1;
  uint32_t *d_total = reinterpret_cast<uint32_t *>(ctx.d_scratch);  // {families, mesh nodes}
  DG_CUDA(cudaMemsetAsync(atab.get(), 0xff, cap * sizeof(uint32_t), s));
  DG_CUDA(cudaMemsetAsync(ctx.d_flags, 0, sizeof(uint32_t), s));
  {
    ProfScope _prof(ctx, "da_leaf_elems", (double)n * 64 + (double)cap * 4);
    k_anchor_insert<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask);
    DG_LAUNCH_CHECK();
    k_mesh_elems<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask, D, ctx.d_etype_of, meta.get(),
                                                  base.get(), ctx.d_flags);
    DG_LAUNCH_CHECK();
    k_family_heads<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask, D, head.get());
    DG_LAUNCH_CHECK();
  }
  exclusive_scan<uint32_t, uint32_t>(head.get(), pos.get(), n, d_total, s);
  exclusive_scan<uint32_t, uint32_t>(base.get(), base.get(), n, d_total + 1, s);
  DG_CUDA(cudaMemcpyAsync(ctx.h_scratch + 4, d_total, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  check_device_flags(ctx, "DA");
  uint32_t total[2];
  std::memcpy(total, ctx.h_scratch + 4, sizeof(total));
  const size_t nf = total[0], nn = total[1], np = (nf + FAM - 1) / FAM;
  if (nn >= (size_t)PRUN_BDY) fail(DG_ERR_INVALID_ARG, "DA: too many nodes for the element loop tables");
  DBuf<uint32_t> conn(8 * n, s), nxyz(3 * (nn ? nn : 1), s), first(nf, s), list(nf, s), state(nf, s),
      lat(np * 27 * FAM, s);
  DBuf<uint2> kids(8 * nf, s);
  {
    ProfScope _prof(ctx, "da_leaf_lattices", (double)n * 72 + (double)nf * 200);
    k_mesh_conn<<<grid_for(n, 256), 256, 0, s>>>(bal.keys, n, atab.get(), amask, D, meta.get(), base.get(),
                                                 conn.get(), nxyz.get(), nxyz.get() + nn, nxyz.get() + 2 * nn, nn,
                                                 ctx.d_flags);
    DG_LAUNCH_CHECK();
    k_family_list<<<grid_for(n, 256), 256, 0, s>>>(head.get(), pos.get(), n, first.get());
    DG_LAUNCH_CHECK();
    k_leaf_lattice<<<(unsigned)np, FAM, 0, s>>>(bal.keys, n, atab.get(), amask, D, first.get(), nf, meta.get(),
                                                conn.get(), list.get(), kids.get(), state.get(), lat.get());
    DG_LAUNCH_CHECK();
  }
  m.n_node = nn;
  m.node_xyz = nxyz.release_ptr();
  if (!m.compressed) m.conn = conn.release_ptr();
  m.meta = meta.release_ptr();
  mesh_patches(ctx, m, list.get(), nf, kids.get(), state.get(), lat.get());
}

void mesh_build(Context &ctx, const Octree &bal, Mesh &m, bool compress) {
  const size_t n = bal.n;
  if (n == 0) fail(DG_ERR_INVALID_ARG, "DA: empty octree");
  if (n >= 0xffffffffull / 8) fail(DG_ERR_INVALID_ARG, "DA: too many elements");
  ensure_stencils(ctx);
  m.max_depth = bal.max_depth;
  m.n_elem = n;
  m.compressed = compress;
  // an octree that came from records: its nodes, if it is one
  struct Made {
    Context &ctx;
    Octree o;
    ~Made() { octree_free(ctx, o); }
  } made{ctx, Octree()};
  try {
    const bool nodes = bal.nodes || octree_nodes(ctx, bal, made.o);
    const Octree &tree = bal.nodes ? bal : made.o;
    if (!nodes) build_from_leaves(ctx, bal, m);
    else if (tree.node_wide) build_from_nodes<Key128>(ctx, bal, tree, m);
    else build_from_nodes<uint64_t>(ctx, bal, tree, m);
  } catch (...) {
    mesh_free(ctx, m);
    throw;
  }
}

void mesh_free(Context &ctx, Mesh &m) {
  if (m.meta) cudaFreeAsync(m.meta, ctx.stream);
  if (m.conn) cudaFreeAsync(m.conn, ctx.stream);
  if (m.node_xyz) cudaFreeAsync(m.node_xyz, ctx.stream);
  if (m.fam) cudaFreeAsync(m.fam, ctx.stream);
  if (m.pinfo) cudaFreeAsync(m.pinfo, ctx.stream);
  if (m.prun) cudaFreeAsync(m.prun, ctx.stream);
  if (m.fchild) cudaFreeAsync(m.fchild, ctx.stream);
  m = Mesh();
}

// ------------------------------------------------------------------------
// element loop
// ------------------------------------------------------------------------
// the element loop's tables for these factors (kept on the context until a call
// with others): the elements' operators per level, and for FP64 vectors the
// fixed-point modes behind them
template <typename T>
static const Cube<T> *cube_table(Context &ctx, double lap_fac, double mass_fac) {
  constexpr bool dbl = std::is_same<T, double>::value;
  Context::CubeTable &t = dbl ? ctx.cubes64 : ctx.cubes32;
  if (!t.p) DG_CUDA(cudaMalloc(&t.p, DTAB_LEVELS * sizeof(Cube<T>) + (dbl ? DTAB_ENTRIES * sizeof(int2) : 0)));
  Cube<T> *p = static_cast<Cube<T> *>(t.p);
  if (!t.ok || t.lap != lap_fac || t.mass != mass_fac) {
    k_cube_table<T><<<1, 32, 0, ctx.stream>>>(p, lap_fac, mass_fac);
    DG_LAUNCH_CHECK();
    if (dbl) {
      k_fix_table<<<(DTAB_ENTRIES + 127) / 128, 128, 0, ctx.stream>>>(reinterpret_cast<int2 *>(p + DTAB_LEVELS),
                                                                      lap_fac, mass_fac);
      DG_LAUNCH_CHECK();
    }
    t.lap = lap_fac;
    t.mass = mass_fac;
    t.ok = true;
  }
  return p;
}

// blocks of a grid-strided patch kernel
template <typename F>
static unsigned patch_grid(Context &ctx, F *kernel, size_t smem, size_t n_patch) {
  ensure_smem_attr(ctx, kernel, 227 * 1024 - 1024);
  int per_sm = 1;
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, FAM, smem));
  return (unsigned)std::min<size_t>(n_patch, (size_t)std::max(per_sm, 1) * ctx.num_sms);
}

template <typename T, bool DIR>
static bool elem_matvec(Context &ctx, const Mesh &m, const uint8_t *bdy, const T *x, T *y, double lap_fac,
                        double mass_fac, const char *name, double bytes) {
  if (!m.conn || m.n_elem > elem_wise_max<T> || (DIR && !bdy)) return false;
  ProfScope _prof(ctx, name, bytes);
  k_elem_matvec<T, DIR><<<grid_for(m.n_elem, 128), 128, 0, ctx.stream>>>(m.meta, m.conn, m.n_elem, bdy, (T)lap_fac,
                                                                         (T)mass_fac, x, y);
  DG_LAUNCH_CHECK();
  return true;
}

template <bool DIR>
void launch_matvec(Context &ctx, const Mesh &m, const uint8_t *bdy, const float *x, float *y, double lap_fac,
                          double mass_fac, const char *name, double bytes) {
  if (elem_matvec<float, DIR>(ctx, m, bdy, x, y, lap_fac, mass_fac, name, bytes)) return;
  const size_t smem = family_smem(m.max_run);
  const unsigned grid = patch_grid(ctx, k_family_matvec<DIR>, smem, m.n_patch);
  const Cube<float> *tab = cube_table<float>(ctx, lap_fac, mass_fac);
  ProfScope _prof(ctx, name, bytes);
  k_family_matvec<DIR><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch, m.max_run, tab,
                                                        x, y);
  DG_LAUNCH_CHECK();
}

template <bool DIR>
void launch_matvec(Context &ctx, const Mesh &m, const uint8_t *bdy, const double *x, double *y,
                          double lap_fac, double mass_fac, const char *name, double bytes) {
  if (elem_matvec<double, DIR>(ctx, m, bdy, x, y, lap_fac, mass_fac, name, bytes)) return;
  const size_t smem = family_fix_smem(m.max_run);
  const unsigned grid = patch_grid(ctx, k_family_matvec_fix<DIR>, smem, m.n_patch);
  const Cube<double> *tab = cube_table<double>(ctx, lap_fac, mass_fac);
  ProfScope _prof(ctx, name, bytes);
  k_family_matvec_fix<DIR><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch, m.max_run,
                                                            reinterpret_cast<const int2 *>(tab + DTAB_LEVELS), tab,
                                                            x, y);
  DG_LAUNCH_CHECK();
}
template void launch_matvec<true>(Context &, const Mesh &, const uint8_t *, const float *, float *, double,
                                         double, const char *, double);
template void launch_matvec<true>(Context &, const Mesh &, const uint8_t *, const double *, double *, double,
                                         double, const char *, double);

template <typename T>
void mesh_matvec(Context &ctx, const Mesh &m, const T *x, T *y, double lap_fac, double mass_fac) {
  DG_CUDA(cudaMemsetAsync(y, 0, m.n_node * sizeof(T), ctx.stream));
  launch_matvec<false>(ctx, m, nullptr, x, y, lap_fac, mass_fac, sizeof(T) == 4 ? "matvec_fp32" : "matvec_fp64",
                              (double)m.n_elem * 36 + (double)m.n_node * 3 * sizeof(T));
}
template void mesh_matvec<float>(Context &, const Mesh &, const float *, float *, double, double);
template void mesh_matvec<double>(Context &, const Mesh &, const double *, double *, double, double);

template <typename T>
void mesh_matvec_coef(Context &ctx, const Mesh &m, const double *coef, const T *x, T *y) {
  DG_CUDA(cudaMemsetAsync(y, 0, m.n_node * sizeof(T), ctx.stream));
  const size_t smem = family_coef_smem<T>(m.max_run);
  const unsigned grid = patch_grid(ctx, k_family_coef<T>, smem, m.n_patch);
  ProfScope _prof(ctx, sizeof(T) == 4 ? "matvec_coef_fp32" : "matvec_coef_fp64",
                  (double)m.n_elem * (36 + 16 + 2) + (double)m.n_node * 3 * sizeof(T));
  k_family_coef<T><<<grid, FAM, smem, ctx.stream>>>(m.fam, m.prun, m.pinfo, m.n_fam, m.n_patch, m.max_run, x, y, coef,
                                                    m.fchild);
  DG_LAUNCH_CHECK();
}
template void mesh_matvec_coef<float>(Context &, const Mesh &, const double *, const float *, float *);
template void mesh_matvec_coef<double>(Context &, const Mesh &, const double *, const double *, double *);

// diagonal entries per element, added atomically (a node's sum is over the
// elements that hold it)
__global__ void k_mesh_diag(const uint32_t *__restrict__ meta, const uint32_t *__restrict__ conn, size_t E,
                            const double *__restrict__ sten, const double *__restrict__ coef, double lap_fac,
                            double mass_fac, double *__restrict__ diag) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const uint32_t me = meta[e];
  const unsigned l = me & 255u, c = (me >> 8) & 7u, t = me >> 24;
  const double h = 1.0 / (double)(1ull << l);
  const double lf = coef ? coef[2 * e] : lap_fac, mf = coef ? coef[2 * e + 1] : mass_fac;
  const double f1 = lf * h / 2.0, f2 = mf * h * h * h / 8.0;
  const double *S = sten + (c * 18 + t) * 128;
#pragma unroll
  for (int k = 0; k < 8; k++) atomicAdd(&diag[conn[(size_t)k * E + e]], f1 * S[9 * k] + f2 * S[64 + 9 * k]);
}

void mesh_diagonal(Context &ctx, const Mesh &m, const double *coef, double lap_fac, double mass_fac, double *diag) {
  ensure_stencils(ctx);
  cudaStream_t s = ctx.stream;
  DG_CUDA(cudaMemsetAsync(diag, 0, m.n_node * sizeof(double), s));
  if (!m.n_elem) return;
  DBuf<uint32_t> tmp;
  const uint32_t *conn = mesh_conn(ctx, m, tmp);
  ProfScope _prof(ctx, "mesh_diagonal", (double)m.n_elem * (4 + 32 + (coef ? 16 : 0)) + (double)m.n_node * 8);
  k_mesh_diag<<<grid_for(m.n_elem, 256), 256, 0, s>>>(m.meta, conn, m.n_elem, ctx.d_sten64, coef, lap_fac, mass_fac,
                                                       diag);
  DG_LAUNCH_CHECK();
}

}  // namespace dg
